// Prefill attention for long prompts on the 5th-generation tensor cores (tcgen05 + TMEM):
// causal / sliding-window softmax(q k^T / 16) v per (query, head), ops::attention_prefill
// (reference ops.hpp:377-526: a sliding-window query s sees keys max(0, s - window) .. s).
//
// The four heads share one KV head, so the (query, head) pairs of 32 consecutive queries form a 128-row
// operand: row r of tile t is query 32 t + r / 4, head r % 4 — the rows of q [S][4][256] as they lie.
// One CTA owns a row tile and walks its keys in tiles of 128:
//     S = Q K_j^T                    M128 x N128, contraction over the 256 head dimensions
//     online softmax on S            (max in use m and sum l per row; a row = one TMEM lane, two threads)
//     O = corr * O + P V_j           M128 x N256, contraction over the tile's keys
// Only the keys that some row of the tile sees are worked on, in units of 16: the first tile of a window and the last one of
// a row tile have a smaller N and fewer V blocks.
// fp32 accuracy on bf16 tensor cores: every fp32 operand is split into three bf16 terms x = hi + mid + lo (all 24 bits, fp32's
// range) and a product a * b is the six term products whose weight reaches
// 2^-24 (hi hi, hi mid, mid hi, mid mid, hi lo, lo hi), all accumulated in fp32 in TMEM.
// Two fp16 terms and three products take less time, but they hold 22 to 23 bits of an
// operand inside fp16's range only, so v would need a scale from keys that a row may not see: its bits, and whether it is finite,
// would hang on later tokens.
//
// Operands are packed once per layer in the tensor core's shared-memory layouts (no swizzle, 8 x 8 core
// matrices), by the kernel that finishes the projections (attn_qkv_pack_kernel), so that the CTA fetches them with plain bulk copies:
//     Q, K: [3 terms][128-row tiles][16 blocks of 16 dimensions][4 KiB], K-major
//     V:    [3 terms][16-key blocks][8 KiB], N-major
// Warps 0-7: softmax and epilogue (two threads per row: warps w and w + 4 share the TMEM lanes 32 (w % 4) ..
// and take half of a tile's keys each); warp 8: one thread issues the MMAs; warp 9: one thread issues the bulk
// copies, up to five ring blocks ahead of the MMAs.
// Per key tile the ring carries 16 Q|K blocks (16 dimensions each) and up to eight V blocks (16 keys each), 24 KiB apiece: Q does
// not fit beside P and the ring and is fetched again for every key tile.
// The tensor pipe bounds it. An MMA of N = 64 takes 48 clk for 32 clk of products, because its 128 rows of A are
// read from shared memory all the same; of N = 128 it takes 64 for 64 (16384 tokens, a sliding-window layer 293 -> 220 us, a global one 3270 -> 2500).
// S is double-buffered in TMEM and the MMAs are issued as Q K_0^T, Q K_1^T, P V_0, Q K_2^T, P V_1, ...: while the
// softmax warps work on tile t the tensor core runs Q K_{t+1}^T and P V_{t-1}. The running max is only moved (and
// O rescaled, a TMEM round trip) when a row's new max exceeds the one in use by more than 8: the probabilities
// are then at most e^8, far inside fp32, and the final division by the row sum removes the common factor.
// The epilogue leaves the digits of the O projection's operand (a row of it is the four heads of a query).
// All waits are bounded; behind one that runs out no copy is issued any more (its stage's barrier may still count an older one), *err is set, and the
// CTA lets its copies land and frees its TMEM before it returns. POLLS, the limit, is 0 in a test (no MMA then
// either); as an argument of the launch it cost 1.4 us a layer.
#pragma once
#include "kernels_gemm_i8.cuh"  // digits of the O projection's operand
#include "kernels_prefill.cuh"  // RopeArgs
#include "kernels_tc.cuh"

namespace tg {

constexpr int AT_TC_BM = 128;                      // rows of a tile: 32 queries x 4 heads
constexpr int AT_TC_KT = 128;                      // keys per tile
constexpr int AT_TC_QBYTES = AT_TC_BM * 16 * 2;    // one term of a Q or K block: [128 rows][16 dimensions] bf16
constexpr int AT_TC_VBYTES = 16 * 256 * 2;         // one term of a V block: [16 keys][256 dimensions] bf16
constexpr int AT_TC_STAGE = 6 * AT_TC_QBYTES;      // ring stage: Q and K blocks (3 x 4 KiB each), or a V block (3 x 8 KiB)
static_assert(AT_TC_STAGE == 3 * AT_TC_VBYTES, "");
constexpr int AT_TC_NS = 5;                        // ring stages
constexpr int AT_TC_PTERM = AT_TC_BM * AT_TC_KT * 2;  // P: one term of [8 blocks of 16 keys][128 rows][16 keys] bf16
constexpr int AT_TC_SMEM = AT_TC_NS * AT_TC_STAGE + 3 * AT_TC_PTERM + 1024;
constexpr int AT_TC_THREADS = 320;                 // 8 softmax warps, the MMA-issuing warp, the copy-issuing warp

// eight fp32 values -> three bf16 terms, one 16-byte store each; every residual is exact
__device__ __forceinline__ void at_split8(__nv_bfloat16 *out, size_t term_stride, const float (&x)[8]) {
	__align__(16) __nv_bfloat16 hi[8], mid[8], lo[8];
#pragma unroll
	for (int i = 0; i < 8; i++) {
		hi[i] = __float2bfloat16_rn(x[i]);
		const float r1 = x[i] - __bfloat162float(hi[i]);
		mid[i] = __float2bfloat16_rn(r1);
		lo[i] = __float2bfloat16_rn(r1 - __bfloat162float(mid[i]));
	}
	*reinterpret_cast<uint4 *>(out) = *reinterpret_cast<const uint4 *>(hi);
	*reinterpret_cast<uint4 *>(out + term_stride) = *reinterpret_cast<const uint4 *>(mid);
	*reinterpret_cast<uint4 *>(out + 2 * term_stride) = *reinterpret_cast<const uint4 *>(lo);
}
__device__ __forceinline__ void at_load8(float (&x)[8], const float *p) {
	const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
	x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}

// The raw sums of the grouped q|k|v GEMM (RopeArgs::part) -> splits added, scaled, q/k norm, RoPE, cache append (as
// qk_norm_rope_prefill_kernel) and the packed operands of the attention, in one pass over memory. 16384 x 1536: 100 us,
// where that kernel, two packing passes over q and k and one over v took 210. (283 MB: 45 us of HBM; four dependent phases at 12 warps per SM bound it.)
// A CTA is 8 positions. A warp does eight rows of the packed operands: warps 0-3 two positions of q with four heads
// each, 4 the keys, 5 the values. Lane (row, quarter) = (lane % 8, lane / 8) holds the dimensions 32 i + 8 * quarter .. + 8, i < 8: a row's sum of squares is two
// shuffles away, RoPE's partner dimension is in the same lane, and a store of the warp fills four core matrices, 512 contiguous bytes (v: whole 128-byte lines).
// Positions >= S are packed as zeros (the tiles of the operands are whole).
__global__ void __launch_bounds__(192) attn_qkv_pack_kernel(RopeArgs a, __nv_bfloat16 *qp, __nv_bfloat16 *kp, __nv_bfloat16 *vp, int q_tiles, int k_tiles,
                                                            int v_blocks) {
	pdl_trigger();
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane & 7, d0 = 8 * (lane >> 3);
	const int p0 = int(blockIdx.x) * 8, s = warp < 4 ? p0 + 2 * warp + (r >> 2) : p0 + r, head = warp < 4 ? r & 3 : 0;
	const int col = warp < 4 ? head * 256 : (warp == 4 ? 1024 : 1280);  // of a row of q | k | v
	const bool in = s < a.S;
	pdl_wait();
	float x[8][8];
	const float *src = a.part + (size_t(blockIdx.y) * a.S + min(s, a.S - 1)) * 1536 + col + d0;
#pragma unroll
	for (int i = 0; i < 8; i++) at_load8(x[i], src + 32 * i);
	for (int sp = 1; sp < a.nsplit; sp++) {
		src += size_t(a.rows) * 1536;
#pragma unroll
		for (int i = 0; i < 8; i++) {
			float y[8];
			at_load8(y, src + 32 * i);
#pragma unroll
			for (int e = 0; e < 8; e++) x[i][e] += y[e];
		}
	}
	const float *sc = (warp < 4 ? a.sq + head * 256 : (warp == 4 ? a.sk : a.sv)) + d0;
#pragma unroll
	for (int i = 0; i < 8; i++) {
		float f[8];
		at_load8(f, sc + 32 * i);
#pragma unroll
		for (int e = 0; e < 8; e++) x[i][e] = in ? x[i][e] * f[e] : 0.0f;
	}
	if (warp < 5) {
		float ss = 0.0f;
#pragma unroll
		for (int i = 0; i < 8; i++)
#pragma unroll
			for (int e = 0; e < 8; e++) ss = fmaf(x[i][e], x[i][e], ss);
		ss += __shfl_xor_sync(0xffffffffu, ss, 8);
		ss += __shfl_xor_sync(0xffffffffu, ss, 16);
		const float rn = inv_rms(ss, 256);
		const float *w = (warp < 4 ? a.rmsq : a.rmsk) + d0;
		const size_t pos = size_t(a.pos0 + min(s, a.S - 1)) * 256 + d0;
#pragma unroll
		for (int i = 0; i < 4; i++) {
			float wl[8], wh[8], cl[8], ch[8], nl[8], nh[8];
			at_load8(wl, w + 32 * i);
			at_load8(wh, w + 128 + 32 * i);
			at_load8(cl, a.cosT + pos + 32 * i);
			at_load8(ch, a.cosT + pos + 128 + 32 * i);
			at_load8(nl, a.sinT + pos + 32 * i);
			at_load8(nh, a.sinT + pos + 128 + 32 * i);
#pragma unroll
			for (int e = 0; e < 8; e++) {
				// y = cos*x + rotate_half(x)*sin, rotate_half = [-x_hi, x_lo]
				const float u = (x[i][e] * rn) * (wl[e] + 1.0f), v = (x[i + 4][e] * rn) * (wh[e] + 1.0f);
				x[i][e] = fmaf(-1.0f * v, nl[e], cl[e] * u);
				x[i + 4][e] = fmaf(u, nh[e], ch[e] * v);
			}
		}
	}
	if (warp >= 4 && in && s >= a.cache_from) {
		float *c = (warp == 4 ? a.kcache : a.vcache) + blockIdx.y * a.cache_stride + size_t((s + a.slot_off) % a.slots) * 256 + d0;
#pragma unroll
		for (int i = 0; i < 8; i++) {
			*reinterpret_cast<float4 *>(c + 32 * i) = make_float4(x[i][0], x[i][1], x[i][2], x[i][3]);
			*reinterpret_cast<float4 *>(c + 32 * i + 4) = make_float4(x[i][4], x[i][5], x[i][6], x[i][7]);
		}
	}
	if (warp < 5) {
		const int tiles = warp < 4 ? q_tiles : k_tiles, row = warp < 4 ? 4 * s + head : s;
		const size_t term = size_t(tiles) * AT_TC_BM * 256;  // elements
		__nv_bfloat16 *out = (warp < 4 ? qp : kp) + blockIdx.y * 3 * term + size_t(row / AT_TC_BM) * (AT_TC_BM * 256) + (row % AT_TC_BM / 8) * 128 + r * 8;
		// dimension 32 i + d0: block 2 i + d0 / 16, 8-wide half (d0 / 8) % 2 of its rows
		const int off = (d0 >> 4) * (AT_TC_QBYTES / 2) + ((d0 >> 3) & 1) * 64;
#pragma unroll
		for (int i = 0; i < 8; i++) at_split8(out + off + i * AT_TC_QBYTES, term, x[i]);
	} else if (s < 16 * v_blocks) {
		const size_t term = size_t(v_blocks) * (AT_TC_VBYTES / 2);
		// (key, dimension n) of a block: (n / 8) * 256 + (key / 8) * 128 + (key % 8) * 16 + (n % 8) * 2 bytes
		__nv_bfloat16 *out = vp + blockIdx.y * 3 * term + size_t(s >> 4) * (AT_TC_VBYTES / 2) + ((s >> 3) & 1) * 64 + r * 8 + (d0 >> 3) * 128;
#pragma unroll
		for (int i = 0; i < 8; i++) at_split8(out + i * 512, term, x[i]);
	}
}

// instruction descriptor: D fp32, A and B bf16, A K-major, B K-major (b_mn = 0) or N-major (1), M = 128, N = n
__device__ __forceinline__ uint32_t at_idesc(int n, int b_mn) {
	return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(b_mn) << 16) | (uint32_t(n >> 3) << 17) | (uint32_t(AT_TC_BM >> 4) << 24);
}
// shared-memory matrix descriptor of a Q, K or P block: K-major, no swizzle, 128 B to the next 8 k, 256 B to the next 8 rows
__device__ __forceinline__ uint64_t at_qdesc(uint32_t smem_addr) {
	return uint64_t((smem_addr & 0x3FFFF) >> 4) | (uint64_t(128 >> 4) << 16) | (uint64_t(256 >> 4) << 32) | (uint64_t(1) << 46);
}
// shared-memory matrix descriptor of a V block: no swizzle, 128 B between the two 8-key groups, 256 B between
// groups of 8 dimensions
__device__ __forceinline__ uint64_t at_vdesc(uint32_t smem_addr) {
	uint64_t d = 0;
	d |= uint64_t((smem_addr & 0x3FFFF) >> 4);
	d |= uint64_t(128 >> 4) << 16;
	d |= uint64_t(256 >> 4) << 32;
	d |= uint64_t(1) << 46;
	return d;
}
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&r)[32]) {
	asm volatile(
	    "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
	    "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
	    "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
	    "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
	    "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
	    : "memory");
}
// Waits of the softmax warps: bounded, given up when another role of the CTA already has, and without an exit: a lane that gave up (ok) goes on with its
// warp and waits no more, since the TMEM loads and stores behind a wait are instructions of the whole, converged warp.
struct AtLimit {
	int polls, *err;
	volatile int *s_fail;
	bool ok = true;
	__device__ __forceinline__ void spin(int &spins) {
		if ((++spins & 1023) == 0 && *s_fail) ok = false;
		if (spins > polls) {
			atomicExch(err, 6);
			*s_fail = 1;
			ok = false;
		}
	}
};
__device__ __forceinline__ void at_wait(uint64_t *bar, uint32_t parity, AtLimit &lim) {
	int spins = 0;
	while (lim.ok && !mbar_try_wait(bar, parity)) lim.spin(spins);
	__syncwarp();
}

// The two threads of a row hand each other one float through shared memory: value, then tag; the reader
// polls the partner's tag (bounded like every wait here).
__device__ __forceinline__ float at_exchange(float *val, int *tag, int me, float v, int t, AtLimit &lim) {
	volatile float *xv = val;
	volatile int *xg = tag;
	xv[me] = v;
	__threadfence_block();
	xg[me] = t;
	int spins = 0;
	while (lim.ok && xg[me ^ 1] != t) lim.spin(spins);
	__syncwarp();
	__threadfence_block();
	return xv[me ^ 1];
}

struct AttnTcArgs {
	// per prompt (blockIdx.y), one behind the other:
	const __nv_bfloat16 *qp;  // [3][q_tiles][16][4 KiB]
	const __nv_bfloat16 *kp;  // [3][k_tiles][16][4 KiB]
	const __nv_bfloat16 *vp;  // [3][v_blocks][8 KiB]
	uint8_t *x;               // digits of the rows [prompts * S][4 * 256] (i8_offset), and their scales
	float *rowscale;
	int groups;
	int S, q_tiles, k_tiles, v_blocks;
	int is_local, window;
	int *err;
};

template <int POLLS>
__global__ void __launch_bounds__(AT_TC_THREADS, 1) attn_prefill_tc_kernel(AttnTcArgs a) {
	pdl_trigger();
	extern __shared__ uint8_t at_smem_raw[];
	uint8_t *smem = reinterpret_cast<uint8_t *>((uintptr_t(at_smem_raw) + 1023) & ~uintptr_t(1023));
	uint8_t *pbuf = smem + AT_TC_NS * AT_TC_STAGE;
	__shared__ uint64_t full_bar[AT_TC_NS];  // the stage's copies landed
	__shared__ uint64_t free_bar[AT_TC_NS];  // the MMAs that read the stage have completed
	__shared__ uint64_t s_bar[2];            // S = Q K^T of a key tile is complete (two S buffers, tiles alternate)
	__shared__ uint64_t p_bar;               // the eight softmax warps wrote P and rescaled O
	__shared__ uint64_t pv_bar;              // P V of a key tile is complete: P may be overwritten, O read
	__shared__ uint64_t o_bar;               // all MMAs done
	__shared__ uint32_t tmem_base_s;
	__shared__ int s_fail;
	__shared__ float xm[2][128][2];          // half-row maxima (by tile parity), row sums at the end
	__shared__ int xt[2][128][2];            // their tags: the exchange between the two threads of a row is a bounded poll

	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int tile = int(gridDim.x) - 1 - int(blockIdx.x);  // the tiles with the most keys start first
	const int q0 = tile * 32;                                // first query of the tile
	const int q_hi = min(a.S - 1, q0 + 31);
	// key tiles this row tile needs, and the blocks of 16 keys of them: u_lo .. 8 of the first, 0 .. u_hi of the last
	const int key_lo = a.is_local ? max(0, q0 - a.window) : 0;
	const int j_lo = key_lo / AT_TC_KT, j_hi = q_hi / AT_TC_KT;
	const int ntiles = j_hi - j_lo + 1;
	const int u_lo = key_lo % AT_TC_KT / 16, u_hi = q_hi % AT_TC_KT / 16 + 1;
	auto first_block = [&](int t) { return t == 0 ? u_lo : 0; };
	auto end_block = [&](int t) { return t == ntiles - 1 ? u_hi : AT_TC_KT / 16; };

	if (tid == 0) {
		for (int s = 0; s < AT_TC_NS; s++) {
			mbar_init(&full_bar[s], 1);
			mbar_init(&free_bar[s], 1);
		}
		mbar_init(&s_bar[0], 1);
		mbar_init(&s_bar[1], 1);
		mbar_init(&p_bar, 8);
		mbar_init(&pv_bar, 1);
		mbar_init(&o_bar, 1);
		s_fail = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	for (int i = tid; i < 2 * 128 * 2; i += AT_TC_THREADS) (&xt[0][0][0])[i] = 0;
	if (warp == 8) {  // TMEM: S in columns 0..127 and 128..255 (alternating tiles), O in columns 256..511
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem_s = tmem_base_s, tmem_o = tmem_base_s + 2u * AT_TC_KT;
	volatile int *fail = &s_fail;

	// Order of the ring blocks and of the MMAs: QK(0), then for t = 1 .. n: QK(t) (if t < n), PV(t - 1)
	auto walk = [&](auto &&qk, auto &&pv) {
		for (int t = 0; t <= ntiles; t++) {
			if (t < ntiles)
				for (int i = 0; i < 16; i++) qk(t, i);  // dimensions 16 i ..
			if (t > 0)
				for (int u = first_block(t - 1); u < end_block(t - 1); u++) pv(t - 1, u);  // keys 16 u ..
		}
	};
	if (warp == 9) {
		// ------------------------------------------------------------ bulk copies, up to AT_TC_NS blocks ahead
		pdl_wait();  // the packed operands are the predecessor's output
		const size_t q_term = size_t(a.q_tiles) * 16 * AT_TC_QBYTES, k_term = size_t(a.k_tiles) * 16 * AT_TC_QBYTES,
		             v_term = size_t(a.v_blocks) * AT_TC_VBYTES;  // bytes
		const uint8_t *qp = reinterpret_cast<const uint8_t *>(a.qp) + blockIdx.y * 3 * q_term + size_t(tile) * 16 * AT_TC_QBYTES,
		              *kp = reinterpret_cast<const uint8_t *>(a.kp) + blockIdx.y * 3 * k_term, *vp = reinterpret_cast<const uint8_t *>(a.vp) + blockIdx.y * 3 * v_term;
		int cap = POLLS, st = 0;
		uint32_t ph = 1;  // (a fresh barrier passes parity 1)
		auto next = [&] {
			if (++st == AT_TC_NS) {
				st = 0;
				ph ^= 1;
			}
		};
		walk(
		    [&](int t, int i) {
			    const uint32_t lo = uint32_t(first_block(t)) * 512u, bytes = uint32_t(end_block(t)) * 512u - lo;  // the block's rows of K: 32 bytes each
			    uint8_t *dst = smem + size_t(st) * AT_TC_STAGE;
			    const uint8_t *q = qp + size_t(i) * AT_TC_QBYTES, *k = kp + (size_t(j_lo + t) * 16 + i) * AT_TC_QBYTES + lo;
			    tc_wait_cap(&free_bar[st], ph, cap);
			    if (tc_elect() && cap > 0) {
				    mbar_expect_tx(&full_bar[st], 3u * (AT_TC_QBYTES + bytes));
#pragma unroll
				    for (int c = 0; c < 3; c++) {
					    bulk_load(dst + c * AT_TC_QBYTES, q + c * q_term, AT_TC_QBYTES, &full_bar[st]);
					    bulk_load(dst + (3 + c) * AT_TC_QBYTES, k + c * k_term, bytes, &full_bar[st]);
				    }
			    }
			    next();
		    },
		    [&](int t, int u) {
			    uint8_t *dst = smem + size_t(st) * AT_TC_STAGE;
			    const uint8_t *v = vp + (size_t(j_lo + t) * (AT_TC_KT / 16) + u) * AT_TC_VBYTES;
			    tc_wait_cap(&free_bar[st], ph, cap);
			    if (tc_elect() && cap > 0) {
				    mbar_expect_tx(&full_bar[st], 3u * AT_TC_VBYTES);
#pragma unroll
				    for (int c = 0; c < 3; c++) bulk_load(dst + c * AT_TC_VBYTES, v + c * v_term, AT_TC_VBYTES, &full_bar[st]);
			    }
			    next();
		    });
		if (cap == 0 && lane == 0) {
			atomicExch(a.err, 6);
			*fail = 1;
		}
	} else if (warp == 8) {
		// ------------------------------------------------------------ MMAs
		const uint32_t idesc_pv = at_idesc(256, 1);
		// the six term products (A term, B term)
		constexpr int ta[6] = {0, 0, 1, 1, 0, 2}, tb[6] = {0, 1, 0, 1, 2, 0};
		int cap = POLLS, st = 0;
		uint32_t ph = 0;
		const uint32_t pb = smem_u32(pbuf);
		bool ready = false;  // the next block has landed: asked before the MMAs of the one before it are issued (an answer takes 180 clk)
		auto landed = [&] {
			if (!ready) tc_wait_cap(&full_bar[st], ph, cap);
			tc_fence_after();
			const int n = st + 1 == AT_TC_NS ? 0 : st + 1;
			ready = mbar_test_wait(&full_bar[n], n ? ph : ph ^ 1u);
			ready = __all_sync(0xffffffffu, ready);
		};
		auto next = [&] {
			__syncwarp();
			if (++st == AT_TC_NS) {
				st = 0;
				ph ^= 1;
			}
		};
		walk(
		    [&](int t, int i) {
			    landed();
			    const uint32_t base = smem_u32(smem + size_t(st) * AT_TC_STAGE), lo = uint32_t(first_block(t)) * 16u, n = uint32_t(end_block(t)) * 16u - lo;
			    const uint32_t d_s = tmem_s + uint32_t(t & 1) * AT_TC_KT + lo, idesc = at_idesc(int(n), 0);
			    const uint64_t dq = at_qdesc(base), dk = at_qdesc(base + 3 * AT_TC_QBYTES);
			    if (POLLS > 0 && tc_elect()) {
#pragma unroll
				    for (int c = 0; c < 6; c++)
					    tc_mma(d_s, dq + uint64_t((ta[c] * AT_TC_QBYTES) >> 4), dk + uint64_t((tb[c] * AT_TC_QBYTES) >> 4), idesc, (i > 0 || c > 0) ? 1u : 0u);
				    tc_commit(&free_bar[st]);
				    if (i == 15) tc_commit(&s_bar[t & 1]);
			    }
			    next();
		    },
		    [&](int t, int u) {
			    if (u == first_block(t)) tc_wait_cap(&p_bar, t & 1, cap);  // P written, O rescaled
			    landed();
			    const uint32_t base = smem_u32(smem + size_t(st) * AT_TC_STAGE);
			    const uint64_t dp = at_qdesc(pb + uint32_t(u) * AT_TC_QBYTES), dv = at_vdesc(base);
			    if (POLLS > 0 && tc_elect()) {
#pragma unroll
				    for (int c = 0; c < 6; c++)
					    tc_mma(tmem_o, dp + uint64_t((ta[c] * AT_TC_PTERM) >> 4), dv + uint64_t((tb[c] * AT_TC_VBYTES) >> 4), idesc_pv,
					           (t > 0 || u > u_lo || c > 0) ? 1u : 0u);
				    tc_commit(&free_bar[st]);
				    if (u == end_block(t) - 1) tc_commit(&pv_bar);
			    }
			    next();
		    });
		if (tc_elect()) tc_commit(&o_bar);
		if (cap == 0 && lane == 0) {
			atomicExch(a.err, 6);
			*fail = 1;
		}
	} else {
		// ------------------------------------------------------------ softmax (two threads per row = TMEM lane)
		// warps w and w + 4 share the TMEM lanes 32 (w % 4) ..: thread (w, lane) owns row 32 (w % 4) + lane and the
		// 64 keys 64 (w / 4) .. of every tile, and half of O's columns
		constexpr int HK = AT_TC_KT / 2;
		const int qd = warp & 3, hf = warp >> 2;
		const int r = qd * 32 + lane;              // row of the tile
		const int qi = q0 + (r >> 2);              // this row's query
		const bool row_ok = qi < a.S;
		const int k_min = a.is_local ? max(0, qi - a.window) : 0;
		const uint32_t lane_base = uint32_t(qd * 32) << 16;
		float m = -INFINITY, l = 0.0f;             // max in use (the same in both threads of a row), sum over this thread's keys
		AtLimit lim{POLLS, a.err, fail};
		for (int jt = 0; jt < ntiles; jt++) {
			at_wait(&s_bar[jt & 1], (jt >> 1) & 1, lim);
			tc_fence_after();
			uint32_t sv[2][32];
			tc_ld32(tmem_s + lane_base + uint32_t((jt & 1) * AT_TC_KT + HK * hf), sv[0]);
			tc_ld32(tmem_s + lane_base + uint32_t((jt & 1) * AT_TC_KT + HK * hf + 32), sv[1]);
			asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
			const int tbase = (j_lo + jt) * AT_TC_KT, kbase = tbase + HK * hf;
			// (most tiles lie wholly inside every row's key range: no per-key test there)
			const bool all_vis = tbase + AT_TC_KT - 1 <= q0 && (!a.is_local || tbase >= q0 + 31 - a.window);
			float mt = -INFINITY;
			if (all_vis) {
#pragma unroll
				for (int c = 0; c < HK; c++) {
					const float x = __uint_as_float(sv[c >> 5][c & 31]) * 0.0625f;  // 1 / sqrt(256), exact
					sv[c >> 5][c & 31] = __float_as_uint(x);
					mt = fmaxf(mt, x);
				}
			} else {  // (columns of keys that no row sees hold nothing: selected away)
#pragma unroll
				for (int c = 0; c < HK; c++) {
					const int key = kbase + c;
					const bool vis = row_ok && key <= qi && key >= k_min;
					const float x = vis ? __uint_as_float(sv[c >> 5][c & 31]) * 0.0625f : -INFINITY;
					sv[c >> 5][c & 31] = __float_as_uint(x);
					mt = fmaxf(mt, x);
				}
			}
			// the row's max over both halves
			mt = fmaxf(mt, at_exchange(xm[jt & 1][r], xt[jt & 1][r], hf, mt, jt + 1, lim));
			// the max in use moves only when the new one exceeds it by more than 8 (or at the row's first visible key)
			const float mn = (mt > m + 8.0f || m == -INFINITY) ? fmaxf(m, mt) : m;
			const bool none = mn == -INFINITY;            // no visible key so far
			const float corr = none ? 1.0f : expf(m - mn);  // exp(-inf) = 0 at the row's first visible tile; 1 when the max stays
			float sum = 0.0f;
#pragma unroll
			for (int c = 0; c < HK; c++) {
				const float p = none ? 0.0f : expf(__uint_as_float(sv[c >> 5][c & 31]) - mn);  // exp(-inf) = 0 for masked keys
				sum += p;
				sv[c >> 5][c & 31] = __float_as_uint(p);
			}
			l = fmaf(l, corr, sum);
			m = mn;
			// the previous tile's P V reads P (and accumulates into O) until pv_bar: wait for it before touching either
			if (jt > 0) at_wait(&pv_bar, (jt - 1) & 1, lim);
			tc_fence_after();
			// the probabilities' three bf16 terms by truncation (p >= 0; hi + mid + lo = p exactly: 8 + 8 + 8 bits), eight keys of the row at a time
#pragma unroll
			for (int k8 = 0; k8 < HK / 8; k8++) {
				uint32_t ph[4], pm[4], pl[4];  // bf16 pairs
#pragma unroll
				for (int c = 0; c < 4; c++) {
					uint32_t hb[2], mb[2], lb[2];
#pragma unroll
					for (int u = 0; u < 2; u++) {
						const int e = 8 * k8 + 2 * c + u;
						const float pv = __uint_as_float(sv[e >> 5][e & 31]);
						hb[u] = __float_as_uint(pv) & 0xFFFF0000u;
						const float r1 = pv - __uint_as_float(hb[u]);
						mb[u] = __float_as_uint(r1) & 0xFFFF0000u;
						lb[u] = __float_as_uint(r1 - __uint_as_float(mb[u]));  // at most 8 significant bits: exact in bf16
					}
					ph[c] = __byte_perm(hb[0], hb[1], 0x7632);
					pm[c] = __byte_perm(mb[0], mb[1], 0x7632);
					pl[c] = __byte_perm(lb[0], lb[1], 0x7632);
				}
				uint8_t *dst = pbuf + (HK / 16 * hf + (k8 >> 1)) * AT_TC_QBYTES + (r >> 3) * 256 + (k8 & 1) * 128 + (r & 7) * 16;
				*reinterpret_cast<uint4 *>(dst) = make_uint4(ph[0], ph[1], ph[2], ph[3]);
				*reinterpret_cast<uint4 *>(dst + AT_TC_PTERM) = make_uint4(pm[0], pm[1], pm[2], pm[3]);
				*reinterpret_cast<uint4 *>(dst + 2 * AT_TC_PTERM) = make_uint4(pl[0], pl[1], pl[2], pl[3]);
			}
			// O = corr * O: this thread's half of the row's 256 columns
			if (jt > 0 && !__all_sync(0xffffffffu, corr == 1.0f)) {
#pragma unroll 1
				for (int c8 = 4 * hf; c8 < 4 * hf + 4; c8++) {
					uint32_t ov[32];
					tc_ld32(tmem_o + lane_base + uint32_t(32 * c8), ov);
					asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
					for (int i = 0; i < 32; i++) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * corr);
					tc_st32(tmem_o + lane_base + uint32_t(32 * c8), ov);
				}
				asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
			}
			fence_proxy_async();  // P: generic-proxy stores -> the tensor core's reads
			tc_fence_before();
			__syncwarp();
			if (lane == 0) mbar_arrive(&p_bar);
		}
		// ------------------------------------------------------------ epilogue: the digits of o = O / l
		// A row of the O projection's operand is the four heads of a query: four neighbouring lanes, in both halves. Its largest value
		// first, then O once more. (The partner is past its last read of a slot: it arrived at p_bar, which o_bar follows.)
		at_wait(&o_bar, 0, lim);
		tc_fence_after();
		const float inv = 1.0f / (l + at_exchange(xm[0][r], xt[0][r], hf, l, 0x40000000, lim));  // (a visible key always exists: the query itself)
		uint32_t mx = 0;
#pragma unroll 1
		for (int c8 = 4 * hf; c8 < 4 * hf + 4; c8++) {
			uint32_t ov[32];
			tc_ld32(tmem_o + lane_base + uint32_t(32 * c8), ov);
			asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
			for (int i = 0; i < 32; i++) mx = max(mx, i8_abs_bits(__uint_as_float(ov[i]) * inv));
		}
		mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
		mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
		mx = max(mx, __float_as_uint(at_exchange(xm[1][r], xt[1][r], hf, __uint_as_float(mx), 0x40000001, lim)));
		const float mul = i8_row_mul(mx);
		const int row = int(blockIdx.y) * a.S + qi, head = r & 3;
		const bool store = row_ok && lim.ok;
		if (store && hf == 0 && head == 0) a.rowscale[row] = i8_row_scale(mx);
#pragma unroll 1
		for (int c8 = 4 * hf; c8 < 4 * hf + 4; c8++) {
			uint32_t ov[32];
			tc_ld32(tmem_o + lane_base + uint32_t(32 * c8), ov);
			asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
			if (store) {
#pragma unroll
				for (int h = 0; h < 2; h++) {  // 16 dimensions: one chunk of 16 bytes per digit
					uint32_t d[4][4];
#pragma unroll
					for (int q = 0; q < 4; q++) {
						uint32_t b[4];
#pragma unroll
						for (int i = 0; i < 4; i++) b[i] = i8_digits(__uint_as_float(ov[16 * h + 4 * q + i]) * inv, mul);
						i8_transpose4(b, d[0][q], d[1][q], d[2][q], d[3][q]);
					}
					uint8_t *p = a.x + i8_offset(row, (head * 256 + 32 * c8 + 16 * h) >> 2, a.groups);
#pragma unroll
					for (int i = 0; i < 4; i++) *reinterpret_cast<uint4 *>(p + 512 * i) = make_uint4(d[i][0], d[i][1], d[i][2], d[i][3]);
				}
			}
		}
	}
	// ---------------------------------------------------------------- teardown
	tc_fence_before();
	__syncthreads();
	if (*fail) {
		// a wait ran out: give the copies and MMAs in flight time to finish before shared memory and TMEM go away
		const long long t0 = clock64();
		while (clock64() - t0 < 2000000) {
		}
		__syncthreads();
	}
	if (warp == 8) {
		__syncwarp();
		tc_fence_after();
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base_s), "r"(512) : "memory");
	}
}

}  // namespace tg
