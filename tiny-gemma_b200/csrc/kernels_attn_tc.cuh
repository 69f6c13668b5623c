// Prefill attention for long prompts on the 5th-generation tensor cores (tcgen05 + TMEM):
// causal / sliding-window softmax(q k^T / 16) v per (query, head), ops::attention_prefill
// (reference ops.hpp:377-526: a sliding-window query s sees keys max(0, s - window) .. s).
//
// The four heads share one KV head, so the (query, head) pairs of 32 consecutive queries form a 128-row
// operand: row r of tile t is query 32 t + r / 4, head r % 4 — the rows of q [S][4][256] as they lie.
// One CTA owns a row tile and walks its keys in tiles of 64:
//     S = Q K_j^T                    M128 x N64, contraction over the 256 head dimensions
//     online softmax on S            (max in use m and sum l per row; a row = one TMEM lane, two threads)
//     O = corr * O + P V_j           M128 x N256, contraction over the 64 keys
// fp32 accuracy on 16-bit tensor cores: every fp32 operand is split into two fp16 terms x = hi + lo, each rounded to
// nearest (11 + 11 significant bits: off by at most 2^-23 of x), and a product a * b is the three term products hi hi, hi lo,
// lo hi, accumulated in fp32 in TMEM. (Three bf16 terms and six products kept 2^-27 of an operand, but every further product is
// a further rounding of the fp32 accumulator, which outweighs both: see the errors at attn_tc_scale.) fp16 has a range of 2^15 to 2^-24: the operands are
// scaled by powers of two that the packing kernels and the attention take from the same place: q and k by the bound that their norm
// weights give, v by the prompt's largest |v| (an atomic maximum in the norm + RoPE kernel), p by 16.
//
// Operands are packed once per layer in the tensor core's shared-memory layouts (no swizzle, 8 x 8 core
// matrices), so that the CTA fetches them with plain bulk copies:
//     Q, K: attn_pack_rows_kernel ([2 terms][128-row tiles][8 blocks of 32 dimensions][8 KiB], K-major; a 64-key
//           tile is one half of a 128-row tile)
//     V:    attn_pack_v_kernel ([2 terms][16-key blocks][8 KiB], N-major like the GEMM's weight operand)
// Two terms of Q (128 KiB) stay in shared memory for the whole walk; with three they were fetched again for every key tile,
// 288 of 384 KB.
// Warps 0-7: softmax and epilogue (two threads per row: warps w and w + 4 share the TMEM lanes 32 (w % 4) ..
// and take half of a tile's keys each); warp 8: one thread issues the MMAs; warp 9: one thread issues the bulk
// copies, up to three ring blocks ahead of the MMAs.
// Per key tile the ring carries four K blocks (64 dimensions each) and four V blocks (16 keys each).
// S is double-buffered in TMEM and the MMAs are issued as Q K_0^T, Q K_1^T, P V_0, Q K_2^T, P V_1, ...: while the
// softmax warps work on tile t the tensor core runs Q K_{t+1}^T and P V_{t-1}. The running max is only moved (and
// O rescaled, a TMEM round trip) when a row's new max exceeds the one in use by more than 8: the probabilities
// are then at most e^8, times 16 inside fp16's range, and the final division by the row sum removes the common factor.
// All waits are bounded; a wait that runs out sets *err, and the CTA lets its copies land and frees its
// TMEM before it returns.
#pragma once
#include "kernels_tc.cuh"

namespace tg {

constexpr int AT_TC_KT = 64;                       // keys per tile
constexpr int AT_TC_STAGE = 16 * 1024;             // ring stage: K (2 terms x 2 blocks of 32 dimensions x 4 KiB), or V (2 x 8 KiB)
constexpr int AT_TC_NS = 3;                        // ring stages
constexpr int AT_TC_QBYTES = 2 * 8 * TC_TILE_BYTES;  // Q: 2 terms x 8 blocks of 32 dimensions
constexpr int AT_TC_PBYTES = 2 * 2 * TC_TILE_BYTES;  // P: 2 terms x 2 blocks of 32 keys x [128][32] fp16
constexpr int AT_TC_SMEM = AT_TC_QBYTES + AT_TC_NS * AT_TC_STAGE + AT_TC_PBYTES + 1024;
constexpr int AT_TC_THREADS = 320;                 // 8 softmax warps, the MMA-issuing warp, the copy-issuing warp
constexpr int AT_TC_BLOCKS = 8;                    // ring blocks per key tile: 4 of K (64 dimensions each), 4 of V (16 keys each)
constexpr int AT_TC_VBYTES = 8192;                 // one term of a V block: [16 keys][256 dimensions] fp16
constexpr float AT_TC_PSCALE = 16.0f;

// ------------------------------------------------------------------ scales
// Against the fp32 kernels (attn_prefill_blk_kernel), keys and values of the layers 1, 5 and the last and logits behind 4001 tokens:
// 270m 3.0e-6, 4.8e-6, 7.0e-6, 8.6e-6 relative, with three bf16 terms and six products 4.2e-6, 5.6e-6, 7.6e-6, 1.09e-5; 1B 2.5e-6, 4.0e-6, 7.6e-6,
// 6.9e-6 against 3.6e-6, 4.8e-6, 9.4e-6, 8.9e-6. Prefill of 16384 tokens 66.1 -> 59.1 ms.
// the power of two that brings a magnitude of at most `bound` to at most 2^13 (RoPE tables of up to 2.8 times the unit circle
// stay inside fp16's 2^16; an element 2^-22 of the bound keeps its 22 bits)
__device__ __forceinline__ float attn_tc_scale(float bound) {
	const int e = int(__float_as_uint(bound) >> 23) - 126;  // bound < 2^e
	return __uint_as_float(uint32_t(max(1, min(253, 127 + 13 - e))) << 23);
}
// Scale of normed and rotated rows of 256: |x| / rms <= 16, the norm's gain 1 + w, sqrt(2) from the rotation. Called by whole warps.
__device__ __forceinline__ float attn_tc_row_scale(const float *w) {
	float m = 0.0f;
#pragma unroll
	for (int i = 0; i < 8; i++) m = fmaxf(m, fabsf(__ldg(w + 32 * i + (threadIdx.x & 31)) + 1.0f));
	return attn_tc_scale(22.7f * warp_max(m));
}
// x * scale as two fp16 terms, pairs of consecutive elements
__device__ __forceinline__ void attn_tc_split(float a, float b, uint32_t &hi, uint32_t &lo) {
	const __half2 h = __floats2half2_rn(a, b);
	const float2 f = __half22float2(h);
	const __half2 l = __floats2half2_rn(a - f.x, b - f.y);  // (the differences are exact)
	hi = *reinterpret_cast<const uint32_t *>(&h);
	lo = *reinterpret_cast<const uint32_t *>(&l);
}
// rows [M][256] (normed by gain 1 + w, rotated) -> [2 terms][m_tiles][8 blocks][8 KiB]; rows >= M are zero. blockIdx.y: the prompt
__global__ void __launch_bounds__(256) attn_pack_rows_kernel(const float *A, const float *w, __half *out, int M, int m_tiles) {
	const float sc = attn_tc_row_scale(w);  // (the weights are nobody's output)
	pdl_trigger();
	pdl_wait();
	A += size_t(blockIdx.y) * M * 256;
	const size_t term_stride = size_t(m_tiles) * 8 * (TC_TILE_BYTES / 2);  // elements
	out += size_t(blockIdx.y) * 2 * term_stride;
	const size_t n_chunks = size_t(m_tiles) * TC_BM * 32;  // one thread per (row, 8 consecutive dimensions)
	for (size_t c = size_t(blockIdx.x) * blockDim.x + threadIdx.x; c < n_chunks; c += size_t(gridDim.x) * blockDim.x) {
		int row, k8;
		tc_chunk_to_row_k8(c, 32, row, k8);
		float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
		if (row < M) {
			a = *reinterpret_cast<const float4 *>(A + size_t(row) * 256 + 8 * k8);
			b = *reinterpret_cast<const float4 *>(A + size_t(row) * 256 + 8 * k8 + 4);
		}
		uint4 hi, lo;
		attn_tc_split(a.x * sc, a.y * sc, hi.x, lo.x);
		attn_tc_split(a.z * sc, a.w * sc, hi.y, lo.y);
		attn_tc_split(b.x * sc, b.y * sc, hi.z, lo.z);
		attn_tc_split(b.z * sc, b.w * sc, hi.w, lo.w);
		const size_t off = (size_t(row / TC_BM) * 8 + (k8 >> 2)) * (TC_TILE_BYTES / 2) + ((row % TC_BM) / 8) * 256 + (k8 & 3) * 64 + (row % 8) * 8;
		*reinterpret_cast<uint4 *>(out + off) = hi;
		*reinterpret_cast<uint4 *>(out + term_stride + off) = lo;
	}
}

// v fp32 [S][256] -> two fp16 terms (scaled by the prompt's largest |v|, vmax) in the N-major operand layout, one 8 KiB tile per 16 keys (one MMA K-step):
// byte offset of (key k, dimension n) = (n / 8) * 256 + (k / 8) * 128 + (k % 8) * 16 + (n % 8) * 2. Keys >= S are zero.
__global__ void __launch_bounds__(256) attn_pack_v_kernel(const float *v, const unsigned *vmax, __half *out, int S, int nblocks) {
	pdl_trigger();
	pdl_wait();
	const float sc = attn_tc_scale(__uint_as_float(vmax[blockIdx.y]));
	v += size_t(blockIdx.y) * S * 256;  // blockIdx.y: the prompt
	out += size_t(blockIdx.y) * 2 * nblocks * 4096;
	const size_t term_stride = size_t(nblocks) * 4096;  // elements
	const size_t n_items = size_t(nblocks) * 16 * 32;   // (key, 8 consecutive dimensions)
	for (size_t c = size_t(blockIdx.x) * blockDim.x + threadIdx.x; c < n_items; c += size_t(gridDim.x) * blockDim.x) {
		const int key = int(c >> 5), n8 = int(c & 31);
		float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
		if (key < S) {
			a = *reinterpret_cast<const float4 *>(v + size_t(key) * 256 + 8 * n8);
			b = *reinterpret_cast<const float4 *>(v + size_t(key) * 256 + 8 * n8 + 4);
		}
		uint4 hi, lo;
		attn_tc_split(a.x * sc, a.y * sc, hi.x, lo.x);
		attn_tc_split(a.z * sc, a.w * sc, hi.y, lo.y);
		attn_tc_split(b.x * sc, b.y * sc, hi.z, lo.z);
		attn_tc_split(b.z * sc, b.w * sc, hi.w, lo.w);
		const int kb = key >> 4, k = key & 15;
		const size_t off = size_t(kb) * 4096 + n8 * 128 + (k >> 3) * 64 + (k & 7) * 8;  // elements
		*reinterpret_cast<uint4 *>(out + off) = hi;
		*reinterpret_cast<uint4 *>(out + term_stride + off) = lo;
	}
}

// instruction descriptor: D fp32, A and B fp16, A K-major, B K-major (b_mn = 0) or N-major (1), M = 128, N = n
__device__ __forceinline__ uint32_t at_idesc(int n, int b_mn) {
	return (1u << 4) | (uint32_t(b_mn) << 16) | (uint32_t(n >> 3) << 17) | (uint32_t(TC_BM >> 4) << 24);
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
// bounded wait that also gives up when another role of the CTA already has
__device__ __forceinline__ bool at_wait(uint64_t *bar, uint32_t parity, int *err, volatile int *s_fail) {
	int spins = 0;
	while (!mbar_try_wait(bar, parity)) {
		if ((++spins & 1023) == 0 && *s_fail) return false;
		if (spins > TC_SPIN_CAP) {
			atomicExch(err, 6);
			*s_fail = 1;
			return false;
		}
	}
	return true;
}

// The two threads of a row hand each other one float through shared memory: value, then tag; the reader
// polls the partner's tag (bounded like every wait here).
__device__ __forceinline__ bool at_exchange(float *val, int *tag, int me, float v, int t, float *other, int *err, volatile int *s_fail) {
	volatile float *xv = val;
	volatile int *xg = tag;
	xv[me] = v;
	__threadfence_block();
	xg[me] = t;
	int spins = 0;
	while (xg[me ^ 1] != t) {
		if ((++spins & 1023) == 0 && *s_fail) return false;
		if (spins > TC_SPIN_CAP) {
			atomicExch(err, 6);
			*s_fail = 1;
			return false;
		}
	}
	__threadfence_block();
	*other = xv[me ^ 1];
	return true;
}

struct AttnTcArgs {
	// per prompt (blockIdx.y), one behind the other:
	const __half *qp;         // [2][q_tiles][8][8 KiB]
	const __half *kp;         // [2][k_tiles][8][8 KiB]
	const __half *vp;         // [2][v_blocks][8 KiB]
	const unsigned *vmax;     // largest |v|, as bits
	const float *rmsq, *rmsk;  // norm weights: the scales of q and k
	float *o;                 // [S][4][256]
	int S, q_tiles, k_tiles, v_blocks;
	int is_local, window;
	int *err;
};

__global__ void __launch_bounds__(AT_TC_THREADS, 1) attn_prefill_tc_kernel(AttnTcArgs a) {
	pdl_trigger();
	extern __shared__ uint8_t at_smem_raw[];
	uint8_t *smem = reinterpret_cast<uint8_t *>((uintptr_t(at_smem_raw) + 1023) & ~uintptr_t(1023));
	uint8_t *qbuf = smem, *ring = smem + AT_TC_QBYTES, *pbuf = ring + AT_TC_NS * AT_TC_STAGE;
	__shared__ uint64_t q_bar;               // Q landed
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
	// key tiles this row tile needs
	const int j_lo = a.is_local ? max(0, q0 - a.window) / AT_TC_KT : 0;
	const int j_hi = q_hi / AT_TC_KT;
	const int ntiles = j_hi - j_lo + 1;

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
		mbar_init(&q_bar, 1);
		s_fail = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	for (int i = tid; i < 2 * 128 * 2; i += AT_TC_THREADS) (&xt[0][0][0])[i] = 0;
	if (warp == 8) {  // TMEM: S in columns 0..63 and 64..127 (alternating tiles), O in columns 128..383
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem_s = tmem_base_s, tmem_o = tmem_base_s + 128u;
	volatile int *fail = &s_fail;

	// MMA order: QK(0), then for t = 1 .. n: QK(t) (if t < n), PV(t - 1). Ring block g in that order:
	// g < 4: QK(0) block g; else g' = g - 4, t = 1 + g' / 8, r = g' % 8: QK(t) block r (r < 4, t < n) or PV(t - 1)
	// block r - 4 (t < n), and the last four blocks are PV(n - 1).
	struct Blk {
		int qk, tile, i;  // qk: 1 = K block i (dimensions 64 i ..) of key tile `tile`, 0 = V block i (keys 16 i ..) of it
	};
	auto blk = [&](int g) -> Blk {
		if (g < 4) return Blk{1, 0, g};
		const int gp = g - 4, t = 1 + gp / AT_TC_BLOCKS, r = gp % AT_TC_BLOCKS;
		if (t >= ntiles) return Blk{0, ntiles - 1, r};
		return r < 4 ? Blk{1, t, r} : Blk{0, t - 1, r - 4};
	};
	const int total = ntiles * AT_TC_BLOCKS;
	if (warp == 9) {
		// ------------------------------------------------------------ bulk copies, up to AT_TC_NS blocks ahead
		pdl_wait();  // the packed operands are the predecessors' output
		const size_t q_term = size_t(a.q_tiles) * 8 * TC_TILE_BYTES, k_term = size_t(a.k_tiles) * 8 * TC_TILE_BYTES,
		             v_term = size_t(a.v_blocks) * AT_TC_VBYTES;  // bytes
		const uint8_t *qp = reinterpret_cast<const uint8_t *>(a.qp) + blockIdx.y * 2 * q_term, *kp = reinterpret_cast<const uint8_t *>(a.kp) + blockIdx.y * 2 * k_term,
		              *vp = reinterpret_cast<const uint8_t *>(a.vp) + blockIdx.y * 2 * v_term;
		if (tc_elect()) {
			mbar_expect_tx(&q_bar, uint32_t(AT_TC_QBYTES));
#pragma unroll
			for (int t = 0; t < 2; t++)
				bulk_load(qbuf + t * 8 * TC_TILE_BYTES, qp + t * q_term + size_t(tile) * 8 * TC_TILE_BYTES, 8 * TC_TILE_BYTES, &q_bar);
		}
		__syncwarp();
		int cap = TC_SPIN_CAP, st = 0;
		uint32_t ph = 1;  // (a fresh barrier passes parity 1)
		for (int g = 0; g < total; g++) {
			const Blk b = blk(g);
			const int j = j_lo + b.tile, i = b.i;
			uint8_t *dst = ring + size_t(st) * AT_TC_STAGE;
			tc_wait_cap(&free_bar[st], ph, cap);
			if (tc_elect()) {
				if (b.qk) {
					mbar_expect_tx(&full_bar[st], uint32_t(AT_TC_STAGE));
#pragma unroll
					for (int t = 0; t < 2; t++)
#pragma unroll
						for (int h = 0; h < 2; h++)
							bulk_load(dst + (2 * t + h) * (TC_TILE_BYTES / 2), kp + t * k_term + (size_t(j >> 1) * 8 + 2 * i + h) * TC_TILE_BYTES + (j & 1) * (TC_TILE_BYTES / 2),
							          TC_TILE_BYTES / 2, &full_bar[st]);
				} else {
					mbar_expect_tx(&full_bar[st], 2u * AT_TC_VBYTES);
#pragma unroll
					for (int t = 0; t < 2; t++)
						bulk_load(dst + t * AT_TC_VBYTES, vp + t * v_term + (size_t(4 * j + i)) * AT_TC_VBYTES, AT_TC_VBYTES, &full_bar[st]);
				}
			}
			if (++st == AT_TC_NS) {
				st = 0;
				ph ^= 1;
			}
		}
		if (cap == 0 && lane == 0) {
			atomicExch(a.err, 6);
			*fail = 1;
		}
	} else if (warp == 8) {
		// ------------------------------------------------------------ MMAs
		const uint32_t idesc_qk = at_idesc(AT_TC_KT, 0), idesc_pv = at_idesc(256, 1);
		// the three term products (A term, B term)
		constexpr int ta[3] = {0, 0, 1}, tb[3] = {0, 1, 0};
		int cap = TC_SPIN_CAP, st = 0;
		uint32_t ph = 0;
		const uint32_t pb = smem_u32(pbuf);
		tc_wait_cap(&q_bar, 0, cap);
		for (int g = 0; g < total; g++) {
			const Blk b = blk(g);
			if (!b.qk && b.i == 0) tc_wait_cap(&p_bar, b.tile & 1, cap);  // P written, O rescaled
			tc_wait_cap(&full_bar[st], ph, cap);
			tc_fence_after();
			const uint32_t base = smem_u32(ring + size_t(st) * AT_TC_STAGE);
			if (b.qk) {
				const uint32_t d_s = tmem_s + uint32_t((b.tile & 1) * AT_TC_KT);
				const uint64_t dq = tc_smem_desc(smem_u32(qbuf) + 2 * b.i * TC_TILE_BYTES), dk = tc_smem_desc(base);
				if (tc_elect()) {
#pragma unroll
					for (int h = 0; h < 2; h++)
#pragma unroll
						for (int c = 0; c < 3; c++)
#pragma unroll
							for (int j2 = 0; j2 < 2; j2++)
								tc_mma(d_s, dq + uint64_t(((8 * ta[c] + h) * TC_TILE_BYTES + j2 * 256) >> 4),
								       dk + uint64_t(((2 * tb[c] + h) * (TC_TILE_BYTES / 2) + j2 * 256) >> 4), idesc_qk, (b.i > 0 || h > 0 || c > 0 || j2 > 0) ? 1u : 0u);
					tc_commit(&free_bar[st]);
					if (b.i == 3) tc_commit(&s_bar[b.tile & 1]);
				}
			} else {
				const int vb = b.i;  // keys 16 vb ..: K-step vb % 2 of P's 32-key block vb / 2
				const uint64_t dp = tc_smem_desc(pb + (vb >> 1) * TC_TILE_BYTES + (vb & 1) * 256), dv = at_vdesc(base);
				if (tc_elect()) {
#pragma unroll
					for (int c = 0; c < 3; c++)
						tc_mma(tmem_o, dp + uint64_t((ta[c] * 2 * TC_TILE_BYTES) >> 4), dv + uint64_t((tb[c] * AT_TC_VBYTES) >> 4), idesc_pv,
						       (b.tile > 0 || vb > 0 || c > 0) ? 1u : 0u);
					tc_commit(&free_bar[st]);
					if (vb == 3) tc_commit(&pv_bar);
				}
			}
			__syncwarp();
			if (++st == AT_TC_NS) {
				st = 0;
				ph ^= 1;
			}
		}
		if (tc_elect()) tc_commit(&o_bar);
		if (cap == 0 && lane == 0) {
			atomicExch(a.err, 6);
			*fail = 1;
		}
	} else {
		// ------------------------------------------------------------ softmax (two threads per row = TMEM lane)
		// warps w and w + 4 share the TMEM lanes 32 (w % 4) ..: thread (w, lane) owns row 32 (w % 4) + lane and the
		// 32 keys 32 (w / 4) .. of every tile (= one of P's two 32-key blocks), and half of O's columns
		const int qd = warp & 3, hf = warp >> 2;
		const int r = qd * 32 + lane;              // row of the tile
		const int qi = q0 + (r >> 2);              // this row's query
		const bool row_ok = qi < a.S;
		const int k_min = a.is_local ? max(0, qi - a.window) : 0;
		const uint32_t lane_base = uint32_t(qd * 32) << 16;
		// S is scaled back (and by 1 / sqrt(256)): powers of two
		const float s_back = 0.0625f / (attn_tc_row_scale(a.rmsq) * attn_tc_row_scale(a.rmsk));
		float m = -INFINITY, l = 0.0f;             // max in use (the same in both threads of a row), sum over this thread's keys
		bool ok = true;
		for (int jt = 0; jt < ntiles && ok; jt++) {
			if (!at_wait(&s_bar[jt & 1], (jt >> 1) & 1, a.err, fail)) { ok = false; break; }
			tc_fence_after();
			uint32_t sv[32];
			tc_ld32(tmem_s + lane_base + uint32_t((jt & 1) * AT_TC_KT + 32 * hf), sv);
			asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
			const int kbase = (j_lo + jt) * AT_TC_KT + 32 * hf;
			// (most tiles lie wholly inside every row's key range: no per-key test there)
			const bool all_vis = (j_lo + jt) * AT_TC_KT + AT_TC_KT - 1 <= q0 && (!a.is_local || (j_lo + jt) * AT_TC_KT >= q0 + 31 - a.window);
			float mt = -INFINITY;
			if (all_vis) {
#pragma unroll
				for (int c = 0; c < 32; c++) {
					const float x = __uint_as_float(sv[c]) * s_back;
					sv[c] = __float_as_uint(x);
					mt = fmaxf(mt, x);
				}
			} else {
#pragma unroll
				for (int c = 0; c < 32; c++) {
					const int key = kbase + c;
					const bool vis = row_ok && key <= qi && key >= k_min;
					const float x = vis ? __uint_as_float(sv[c]) * s_back : -INFINITY;
					sv[c] = __float_as_uint(x);
					mt = fmaxf(mt, x);
				}
			}
			// the row's max over both halves
			{
				float other;
				if (!at_exchange(xm[jt & 1][r], xt[jt & 1][r], hf, mt, jt + 1, &other, a.err, fail)) { ok = false; break; }
				mt = fmaxf(mt, other);
			}
			// the max in use moves only when the new one exceeds it by more than 8 (or at the row's first visible key)
			const float mn = (mt > m + 8.0f || m == -INFINITY) ? fmaxf(m, mt) : m;
			const bool none = mn == -INFINITY;            // no visible key so far
			const float corr = none ? 1.0f : expf(m - mn);  // exp(-inf) = 0 at the row's first visible tile; 1 when the max stays
			// probabilities and their two fp16 terms
			float sum = 0.0f;
			uint32_t ph[16], pl[16];  // fp16 pairs
#pragma unroll
			for (int c = 0; c < 32; c += 2) {
				const float p0 = none ? 0.0f : expf(__uint_as_float(sv[c]) - mn), p1 = none ? 0.0f : expf(__uint_as_float(sv[c + 1]) - mn);  // exp(-inf) = 0 for masked keys
				sum += p0;
				sum += p1;
				attn_tc_split(p0 * AT_TC_PSCALE, p1 * AT_TC_PSCALE, ph[c / 2], pl[c / 2]);
			}
			l = fmaf(l, corr, sum);
			m = mn;
			// the previous tile's P V reads P (and accumulates into O) until pv_bar: wait for it before touching either
			if (jt > 0 && !at_wait(&pv_bar, (jt - 1) & 1, a.err, fail)) { ok = false; break; }
			tc_fence_after();
			// P[term][block hf] tiles of [128][32] in the A-operand layout
#pragma unroll
			for (int k8 = 0; k8 < 4; k8++) {
				uint8_t *dst = pbuf + hf * TC_TILE_BYTES + (r >> 3) * 512 + k8 * 128 + (r & 7) * 16;
				*reinterpret_cast<uint4 *>(dst) = make_uint4(ph[4 * k8], ph[4 * k8 + 1], ph[4 * k8 + 2], ph[4 * k8 + 3]);
				*reinterpret_cast<uint4 *>(dst + 2 * TC_TILE_BYTES) = make_uint4(pl[4 * k8], pl[4 * k8 + 1], pl[4 * k8 + 2], pl[4 * k8 + 3]);
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
		// ------------------------------------------------------------ epilogue: o = O / l
		if (ok && at_wait(&o_bar, 0, a.err, fail)) {
			tc_fence_after();
			pdl_wait();  // (vmax; long satisfied)
			float l_other = 0.0f;  // (the partner is past its last read of slot 0: it arrived at p_bar, which o_bar follows)
			const bool got = at_exchange(xm[0][r], xt[0][r], hf, l, 0x40000000, &l_other, a.err, fail);
			const float lt = l + l_other;
			const float inv = (row_ok && got) ? 1.0f / (lt * (AT_TC_PSCALE * attn_tc_scale(__uint_as_float(a.vmax[blockIdx.y])))) : 0.0f;  // (a visible key always exists: the query itself)
			float *orow = a.o + (size_t(blockIdx.y) * a.S * 4 + size_t(tile) * 128 + r) * 256;
#pragma unroll 1
			for (int c8 = 4 * hf; c8 < 4 * hf + 4; c8++) {
				uint32_t ov[32];
				tc_ld32(tmem_o + lane_base + uint32_t(32 * c8), ov);
				asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
				if (row_ok) {
#pragma unroll
					for (int i = 0; i < 32; i += 4)
						*reinterpret_cast<float4 *>(orow + 32 * c8 + i) =
						    make_float4(__uint_as_float(ov[i]) * inv, __uint_as_float(ov[i + 1]) * inv, __uint_as_float(ov[i + 2]) * inv,
						                __uint_as_float(ov[i + 3]) * inv);
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
