// Persistent decode kernel: the whole per-token forward (and the sampler) of one
// sequence in ONE cooperative launch, one CTA per SM, 12 warps per CTA.
//
// At batch 1 a Gemma-3-1B layer is 26.8 MB of int8 weights — 4 us of HBM time —
// spread over five dependent phases, so the time of a token is the length of
// that dependency chain, not the data movement. The design therefore
//   * streams weights a layer ahead: every CTA owns a fixed unit of each weight
//     matrix (column groups x K-range), stored contiguously in a re-tiled copy,
//     and fetches it with bulk copies (cp.async.bulk) into a shared-memory
//     region reserved for that phase. A region is refilled for the NEXT layer
//     as soon as its last reader is done, so about one layer of weights per SM
//     is always in flight and HBM never waits for the chain;
//   * multiplies on the tensor cores (tcgen05.mma kind::i8), from the shared memory the weights land in. The
//     activation vector is quantised once per phase to 31-bit block fixed point (four signed 8-bit digits, one
//     power-of-two exponent per vector); weight columns are the M rows of the operation and the digits its N
//     columns, so the integer sums are exact. One vector would use 4 of 16 columns and a unit of 16 weight columns
//     16 of 64 rows: the K range of a unit is cut into segments that sit side by side as further rows (weights) and
//     columns (digits); the products of equal segments are the ones that are read back, and added as integers;
//   * hands results over through small L2-resident vectors that validate
//     themselves (a sentinel marks words not yet written). Polled bytes are the
//     cost of a hand-off (about 40 ns per KB and CTA), so producers publish
//     final, scaled values wherever a consumer would otherwise re-add K-split
//     partial sums;
//   * recomputes RMSNorms redundantly in every CTA from those vectors; the
//     residual stream lives in each CTA's shared memory.
//
// Phases per layer (reference modules.hpp:135-169, 203-220):
//   A  residual + post-norm of the previous MLP, pre-norm, Q|K|V  -> q|k|v
//   B  q/k norm, RoPE, KV append, attention: CTA = (head, chunk of the cache)
//                                                    -> (m, l, o) per chunk
//   C  merge of the chunks of one head, O projection -> partial sums per head
//   D  residual + post-norm, pre-norm, up & gate, LUT-GeGLU -> activations
//   E  down projection                               -> partial sums per split
// then the lm_head (streamed through a ring of bulk copies from a re-tiled
// copy) and the sampler (argmax, or min-p with the sequential fp32 inverse CDF
// of reference ops.hpp:848-858 evaluated by an exact scan).
//
// Arithmetic: y[n] = scale[n] * sum_k x[k] W[k,n] (reference linalg.hpp:41-204)
// with x rounded to a multiple of 2^-30 of the power of two above the largest
// |x| of the vector (fp32 itself keeps 24 bits relative to each element); products
// and sums are exact, one rounding when the integer sum becomes a float.
//
// Every wait is bounded: a spin that runs out sets *err and a shared abort
// flag, after which all waits fall through and the kernel returns.
#pragma once
#include <cuda.h>

#include "kernels_decode.cuh"
#include "kernels_gemm_i8.cuh"  // digits, tcgen05 helpers
#include "kernels_sampler.cuh"
#include "persist_plan.h"  // units and their tiles
#include "tg_common.cuh"

namespace tg {

constexpr int PS_MAX_LAYERS = 32;
constexpr int PS_MAX_CH = 32;            // most cache chunks per head
constexpr int PS_ATT_ROW = AT_HD + 8;    // floats per attention partial: o[256], m, l, padding
constexpr uint32_t PS_BULK_PIECE = 16384;
constexpr unsigned PS_EMPTY = 0xFFFFFFFFu;  // "not written yet": a NaN no computation produces

constexpr int PS_TMEM = 64;              // TMEM columns: 16 per tile of a unit, or two accumulators of the lm_head
constexpr int PS_ACT = 3;                // quads of a thread in the down projection's prologue, at most
constexpr int PS_LUT = 1024;             // largest GeLU table that is kept in shared memory

struct PsLayer {
	const float *rmsq, *rmsk, *attn_pre, *attn_post, *mlp_pre, *mlp_post;
	float *kcache, *vcache;
	int slots, is_local;
};

// where a token stands in the caches of the sliding-window or of the global layers
struct PsSpan {
	int p, slot, valid;  // position, slot of its row, rows to attend to
	int nch, chunk;      // cache chunks per head, rows of a chunk
};
struct PsArgs {
	const int8_t *tiled;  // re-tiled layer weights: per layer [A units | C units | D units (up, gate) | E units]
	size_t tl_layer, tl_A, tl_C, tl_D, tl_E;
	const int8_t *lm_tiled;  // re-tiled lm_head: [tile][chunk] ring stages of core matrices
	const PsLayer *layers;
	int L, D, I, V, QD, KD;
	PsPhase A, C, Dp, E;
	// lm_head: column tiles of 128 columns; a tile's rows arrive as lm_nchunk ring stages of lm_steps * 32 rows
	int lm_steps, lm_nchunk, lm_ntiles, lm_stages, lm_stage_bytes, lm_pre;
	PsPhase lm;  // (the digits' layout: one segment)
	const float *lm_scale, *final_norm;
	const int8_t *wte;
	const float *wte_s;
	float sqrtD;
	const float *rope[2][2];  // [is_local][cos, sin]
	GeluLut lut;
	int off_A, off_C, off_D, off_E, off_h, off_att, off_lut, smem_total;
	// Hand-off arena, three copies used by consecutive layers; every float is PS_EMPTY or a value.
	//   ll_qkv [QD + 2 KD]                 q|k|v, scaled                      (A -> B)
	//   ll_att [4][PS_MAX_CH][PS_ATT_ROW]  attention partials per head, chunk (B -> C)
	//   ll_op  [C.nsplit][D]               O projection, scaled partial sums  (C -> D)
	//   ll_act [I]                         GeGLU activations                  (D -> E)
	//   ll_dn  [E.nsplit][D] + presence    down projection, scaled partials   (E -> A of the next layer);
	//                                      one presence word for every CTA without a down unit
	float *ll;
	int ll_stride, ll_qkv, ll_att, ll_op, ll_act, ll_dn, ll_pres;
	uint32_t piece_D, piece_E;  // bytes of a quarter of an up/gate and of a down unit
	int merge_heads;  // heads whose attention output an O unit multiplies (4 / C.nsplit)
	int nch_max, nch_local, nch_global;  // cache chunks per head: at most; a number given for sliding-window and global layers (0: by rule)
	int slots_local, slots_global;
	float *logits;
	float *probs;
	float *samp_f;
	int *samp_i;
	float *xnorm_out;
	unsigned *bar;          // grid-barrier counter: bar_base arrivals so far (it is never reset between launches)
	unsigned bar_base;
	int *err;
	int *tok, *next_pos, *ring_base, *tok_log, *log_count;
	int log_cap, n_steps, sampler;
	const int *force_ids;  // optional [n_steps]: the token of every step is given (continuation of a context), not sampled
	float minp, temp;
	const float *randf;
	int *randf_count;
	int randf_cap;
	long long *dbg;
	int dbg_cta, dbg_cap;
	long long wait_clocks;  // SM clocks before a wait gives up
	int poll_ns;            // sleep between two rounds of a hand-off poll
	long long *gt;  // optional: [CTA][12] global-timer marks of one layer (DBG instantiation)
	int *beacon;    // optional (mapped host memory): [CTA][16] progress marks of every warp, for diagnosing a stall
	int fault_cta;  // test hook: this CTA withholds its down-projection hand-off (-1: none); the waits then run out
};

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t ps_smem(const void *p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void ps_mbar_init(uint64_t *bar, int count) {
	asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(ps_smem(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void ps_mbar_expect(uint64_t *bar, uint32_t bytes) {
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(ps_smem(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ps_mbar_arrive(uint64_t *bar) {
	asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(ps_smem(bar)) : "memory");
}
__device__ __forceinline__ bool ps_mbar_try(uint64_t *bar, uint32_t parity) {
	uint32_t ok;
	asm volatile(
	    "{\n\t.reg .pred p;\n\t"
	    "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
	    "selp.u32 %0, 1, 0, p;\n\t}"
	    : "=r"(ok)
	    : "r"(ps_smem(bar)), "r"(parity)
	    : "memory");
	return ok != 0;
}
// Weights are read once per token: evict-first keeps the L2 for the KV cache and the hand-off vectors.
__device__ __forceinline__ uint64_t ps_evict_first() {
	uint64_t pol;
	asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
	return pol;
}
// Untiled bulk copy global -> this CTA's shared memory, completing on an mbarrier (never cluster-wide).
__device__ __forceinline__ void ps_bulk(void *dst, const void *src, uint32_t bytes, uint64_t *bar, uint64_t pol) {
	asm volatile(
	    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(ps_smem(dst)),
	    "l"(src), "r"(bytes), "r"(ps_smem(bar)), "l"(pol)
	    : "memory");
}
// Small vectors that every token reads again (column scales, norm weights, RoPE rows): kept in the L2
// (evict-last) so that they are L2 hits while the weight stream (evict-first) passes through.
__device__ __forceinline__ uint64_t ps_evict_last() {
	uint64_t pol;
	asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
	return pol;
}
__device__ __forceinline__ float ps_ldk(const float *p, uint64_t keep) {
	float v;
	asm volatile("ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(keep));
	return v;
}
__device__ __forceinline__ float4 ps_ldk4(const float *p, uint64_t keep) {
	float4 v;
	asm volatile("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p), "l"(keep));
	return v;
}
__device__ __forceinline__ void ps_fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void ps_prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ unsigned ps_ld_acquire(const unsigned *p) {
	unsigned v;
	asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
	return v;
}
__device__ __forceinline__ void ps_st(float *p, float v) { asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory"); }
__device__ __forceinline__ float4 ps_ld4(const float *p) {
	float4 r;
	asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "l"(p) : "memory");
	return r;
}
__device__ __forceinline__ float2 ps_ld2(const float *p) {
	float2 r;
	asm volatile("ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];" : "=f"(r.x), "=f"(r.y) : "l"(p) : "memory");
	return r;
}
__device__ __forceinline__ float ps_ld1(const float *p) {
	float r;
	asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(r) : "l"(p) : "memory");
	return r;
}
__device__ __forceinline__ bool ps_ok(float v) { return __float_as_uint(v) != PS_EMPTY; }
__device__ __forceinline__ bool ps_ok(const float2 &v) { return ps_ok(v.x) && ps_ok(v.y); }
__device__ __forceinline__ bool ps_ok(const float4 &v) { return ps_ok(v.x) && ps_ok(v.y) && ps_ok(v.z) && ps_ok(v.w); }
// What a wait needs to know to give up: the CTA's abort flag, the global error word, the time limit.
struct PsW {
	int *s_abort;
	int *err;
	long long limit;  // SM clocks a wait may take
	unsigned nap;     // nanoseconds a poller sleeps between rounds
};
__device__ __forceinline__ bool ps_mbar_test(uint64_t *bar, uint32_t parity) {
	uint32_t ok;
	asm volatile(
	    "{\n\t.reg .pred p;\n\t"
	    "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
	    "selp.u32 %0, 1, 0, p;\n\t}"
	    : "=r"(ok)
	    : "r"(ps_smem(bar)), "r"(parity)
	    : "memory");
	return ok != 0;
}
// Give up: the first error code wins (code in the low byte, `where` = layer << 4 | phase above it);
// every later wait of this CTA falls through.
__device__ __noinline__ void ps_give_up(int *s_abort, int *err, int code) {
	*s_abort = 1;
	atomicCAS(err, 0, code);
}
// Wait for a bulk-copy barrier: non-blocking test in a loop bounded by the clock (the blocking
// try_wait form may suspend a thread for an unspecified time per call).
__device__ __noinline__ void ps_wait_bulk_slow(const PsW w, int where, uint64_t *bar, uint32_t parity) {
	const long long t0 = clock64();
	int spins = 0;
	while (!ps_mbar_test(bar, parity)) {
		if ((++spins & 63) == 0 && (clock64() - t0 > w.limit || *(volatile int *)w.s_abort)) {
			ps_give_up(w.s_abort, w.err, 3 | (where << 8));
			return;
		}
	}
}
__device__ __forceinline__ void ps_wait_bulk(const PsW &w, int where, uint64_t *bar, uint32_t parity) {
	if (*(volatile int *)w.s_abort) return;
	if (!ps_mbar_test(bar, parity)) ps_wait_bulk_slow(w, where, bar, parity);
}
// One more round of a hand-off poll? Gives up when the wait has taken w.limit clocks; a CTA that
// gave up (or saw the global error word) lets every later wait fall through.
__device__ __noinline__ bool ps_retry_slow(const PsW w, int where, long long t0) {
	if (clock64() - t0 > w.limit || *(volatile int *)w.err != 0) {
		ps_give_up(w.s_abort, w.err, 5 | (where << 8));
		return false;
	}
	return true;
}
__device__ __forceinline__ bool ps_retry(const PsW &w, int where, int &spins, long long &t0) {
	if (*(volatile int *)w.s_abort) return false;
	if (spins == 0) t0 = clock64();
	if ((++spins & 15) == 0 && !ps_retry_slow(w, where, t0)) return false;
	__nanosleep(w.nap);
	return true;
}

// grid-wide barrier: one atomic counter, bounded spin
__device__ __noinline__ void ps_grid_sync(const PsW w, int where, unsigned *bar, unsigned target) {
	__syncthreads();
	if (threadIdx.x == 0) {
		__threadfence();
		const unsigned old = atomicAdd(bar, 1u);
		// (the counter runs on from launch to launch and may wrap: compare differences, not values)
		if (old + 1u != target && !*(volatile int *)w.s_abort) {  // the last arriver need not poll
			const long long t0 = clock64();
			int spins = 0;
			while (int(ps_ld_acquire(bar) - target) < 0) {
				if ((++spins & 15) == 0 && clock64() - t0 > w.limit) {
					ps_give_up(w.s_abort, w.err, 4 | (where << 8));
					break;
				}
			}
		}
	}
	__syncthreads();
}

// ------------------------------------------------------------------ shared memory by 32-bit shared-window address
// (The helpers below are not inlined, so a pointer argument would be a generic pointer and every access a generic one.)
__device__ __forceinline__ uint4 ps_lds128(uint32_t addr) {
	uint4 v;
	asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
	return v;
}
__device__ __forceinline__ float ps_ldsf(uint32_t addr) {
	float v;
	asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
	return v;
}
__device__ __forceinline__ void ps_stsf(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }

// ------------------------------------------------------------------ quantised activations
// What a phase's unit fixes for the whole launch, in shared memory: a field read from the kernel's arguments costs a
// constant-cache miss where a layer's code has passed through the caches since, and a value kept in a register across the calls
// of a layer is spilled.
struct PsUnit {
	uint64_t da[PS_TILES], db[PS_TILES];  // descriptors of a tile's first MMA: weights, digits
	int tiles, steps, mt;
	uint32_t x_s, seg_mul;  // digits: shared-window address and layout
	int seg_q, x_sbo;
	uint32_t acc_s, scale_s;  // column sums, column scales (behind the unit's weights)
	int rows, segs, ncol, two;
	int dst;           // where the unit's columns go in a copy of the hand-off arena
	int ep[PS_NW];     // per warp: accumulator column | (first entry of the column sums) << 8
};
// A vector x[0..4 nq) becomes the digits of round(x * 2^(30 - e)), 2^e > max |x|: q = d0 + 256 d1 + 65536 d2 + 2^24 d3 with
// d_i in [-128, 127] (the digits of the prefill's GEMM).
__device__ __forceinline__ uint32_t ps_xaddr(const PsUnit *u, int q) { return u->x_s + uint32_t(ps_digit_offset(u->seg_mul, u->seg_q, u->x_sbo, q)); }
// exponent for a bound on max |x| (clamped so that both scale factors are normal floats); a vector with an infinity gives NaN
__device__ __forceinline__ int ps_exponent(float bound) { return max(-96, min(100, (int(__float_as_uint(bound) >> 23) & 0xFF) - 126)); }
__device__ __forceinline__ float ps_pow2(int e) { return __uint_as_float(uint32_t(e + 127) << 23); }
__device__ __forceinline__ float ps_qmul(float M) { return ps_pow2(30 - ps_exponent(M * 1.000001f)); }
__device__ __forceinline__ float ps_qscale(float M) { return M < INFINITY ? ps_pow2(ps_exponent(M * 1.000001f) - 30) : __uint_as_float(0x7FC00000u); }
__device__ __forceinline__ void ps_sts32(uint32_t addr, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
// four elements at p = ps_xaddr(u, quad). (Lanes of a warp hold consecutive quads: four words of a 16-byte chunk, chunks 36 words
// apart: no bank conflict.)
__device__ __forceinline__ void ps_quantise(float4 y, float mul, uint32_t p) {
	const uint32_t a = i8_digits(y.x, mul), b = i8_digits(y.y, mul), c = i8_digits(y.z, mul), d = i8_digits(y.w, mul);
	const uint32_t ab01 = __byte_perm(a, b, 0x5140), ab23 = __byte_perm(a, b, 0x7362);
	const uint32_t cd01 = __byte_perm(c, d, 0x5140), cd23 = __byte_perm(c, d, 0x7362);
	ps_sts32(p, __byte_perm(ab01, cd01, 0x5410));
	ps_sts32(p + 16, __byte_perm(ab01, cd01, 0x7632));
	ps_sts32(p + 32, __byte_perm(ab23, cd23, 0x5410));
	ps_sts32(p + 48, __byte_perm(ab23, cd23, 0x7632));
}
// maximum of non-negative floats over a warp: their bit patterns order like the values
__device__ __forceinline__ float ps_warp_max(float v) { return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v))); }
// the PS_NW floats at p (16-byte aligned): sum in index order, maximum
__device__ __forceinline__ void ps_lds12(uint32_t p, float (&v)[PS_NW]) {
#pragma unroll
	for (int i = 0; i < PS_NW; i += 4)
		asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[i]), "=f"(v[i + 1]), "=f"(v[i + 2]), "=f"(v[i + 3]) : "r"(p + 4u * i) : "memory");
}
__device__ __forceinline__ float ps_sum12(uint32_t p) {
	float v[PS_NW];
	ps_lds12(p, v);
	float t = v[0];
#pragma unroll
	for (int i = 1; i < PS_NW; i++) t += v[i];
	return t;
}
__device__ __forceinline__ float ps_max12(uint32_t p) {
	float v[PS_NW];
	ps_lds12(p, v);
	float t = v[0];
#pragma unroll
	for (int i = 1; i < PS_NW; i++) t = fmaxf(t, v[i]);
	return t;
}
// max over the CTA of a non-negative value through `red` (PS_NW floats; one barrier)
__device__ __forceinline__ float ps_block_max(float mx, float *red) {
	mx = ps_warp_max(mx);
	if ((threadIdx.x & 31) == 0) ps_stsf(ps_smem(red + (threadIdx.x >> 5)), mx);
	__syncthreads();
	return ps_max12(ps_smem(red));
}

// ------------------------------------------------------------------ unit products
__device__ __forceinline__ uint64_t ps_desc(uint32_t addr, int lbo, int sbo) {  // K-major operand without swizzle
	return uint64_t((addr & 0x3FFFF) >> 4) | (uint64_t(lbo >> 4) << 16) | (uint64_t(sbo >> 4) << 32) | (uint64_t(1) << 46);
}
__device__ __forceinline__ uint32_t ps_idesc(int mt) {  // D int32, A and B signed 8 bit, both K-major, M = mt, N = 16
	return (2u << 4) | (1u << 7) | (1u << 10) | (2u << 17) | (uint32_t(mt >> 4) << 24);
}
__device__ __forceinline__ int4 ps_tmem_ld4(uint32_t taddr) {  // 32 lanes x 4 columns
	int4 v;
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(taddr) : "memory");
	asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
	return v;
}
// sum of digit sum i * 256^i, exact (at most 2^30 * 127 * 6912 < 2^50), rounded once
__device__ __forceinline__ float ps_join(const int4 &s) {
	return __ll2float_rn((((((long long)s.w << 8) + s.z) << 8) + s.y) * 256ll + s.x);
}
// what a CTA's place in the grid fixes for the whole launch (kept in shared memory, read where it is used)
struct PsCta {
	const int8_t *srcA, *srcC, *srcD, *srcE;
	uint64_t policy_first, policy_last;  // L2 evict-first (weights) and evict-last (what every token reads again)
	int splitC, splitE, presE, has;
	uint32_t tm;  // TMEM base (the word that tcgen05.alloc wrote, which the compiler does not see written: read once, volatile)
};
// what one token leaves to the next (in shared memory, written by thread 0 between barriers: a register that lives across the
// calls of a layer is spilled, and the L1 beside 224 KB of shared memory does not hold the spills)
struct PsLive {
	uint32_t plm, pemp, acc_n;  // lm_head: parities of the ring's barriers, tiles so far
	unsigned epoch;             // grid barriers passed
	int n_logged, tok, pos;
};
// fields of a phase's entry; `warp` fills its own
__device__ __noinline__ void ps_fill_unit(const PsPhase &ph, PsUnit *u, int warp, uint32_t smem_s, int off_tile, int dst) {
	const int t = warp >> 2;
	if (t < ph.tiles) {
		int r0, col;
		ps_warp_rows(ph, warp, r0, col);
		u->ep[warp] = (16 * t + col) | (r0 << 8);
	}
	if (warp == 0) {
#pragma unroll
		for (int i = 0; i < PS_TILES; i++) {
			u->da[i] = ps_desc(smem_s + uint32_t(off_tile + i * ph.steps * ph.mt * 32), ph.mt * 16, 128);
			u->db[i] = ps_desc(smem_s + uint32_t(ph.off_x + (ps_tile_segment(ph.rows, ph.mt, i) / 2) * ph.x_sbo), PS_XCH, ph.x_sbo);
		}
		u->tiles = ph.tiles;
		u->steps = ph.steps;
		u->mt = ph.mt;
		u->x_s = smem_s + uint32_t(ph.off_x);
		u->seg_mul = ph.seg_mul;
		u->seg_q = ph.seg_q;
		u->x_sbo = ph.x_sbo;
		u->acc_s = smem_s + uint32_t(ph.off_acc);
		u->scale_s = smem_s + uint32_t(off_tile + ph.rows * ph.nq * 4);
		u->rows = ph.rows;
		u->segs = ph.segs;
		u->ncol = ph.ncol;
		u->two = ph.nmat == 2;
		u->dst = dst;
	}
}
// lut::GeLUTable::lookup (reference ops.hpp:41-51); tab_s: the table in shared memory where it fits there
__device__ __forceinline__ float ps_gelu(const GeluLut &t, float x, uint32_t tab_s, uint64_t keep) {
	int idx;
	if (!t.index(x, idx)) return 0.0f;
	if (idx >= t.size) return x;
	return t.size <= PS_LUT ? ps_ldsf(tab_s + 4u * idx) : ps_ldk(t.table + idx, keep);
}
// What a thread needs for its part of a unit's product, fetched before the phase's prologue polls: behind the prologue every
// shared-memory access counts (~30 clk, five of them in a row before the first MMA).
struct PsRun {
	uint64_t da, db;          // issuing warps: descriptors of the first MMA
	uint32_t d, taddr, acc;   // accumulator; where this warp's sums are and go
	int steps, mt;            // steps: 0 where this warp's tile does not exist
	uint32_t col;             // this thread's column: sums of its first segment
	int cstep, segs, ncol, two;
	float s0, s1;             // its scales
};
// The issuing warps, and the ones that read column scales, wait for the unit here (a completed test takes ~200 clk).
__device__ __forceinline__ PsRun ps_prepare(const PsW &w, int where, const PsUnit *u, uint32_t tmem, uint64_t *bar_w, uint32_t pw) {
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, t = warp >> 2;
	PsRun r;
	r.ncol = u->ncol;
	if ((warp & 3) == 0 || 32 * warp < r.ncol) ps_wait_bulk(w, where, bar_w, pw);
	r.da = u->da[t];
	r.db = u->db[t];
	r.d = tmem + 16u * t;
	r.mt = u->mt;
	r.steps = t < u->tiles ? u->steps : 0;
	const int m = u->ep[warp];
	r.taddr = tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(m & 0xFF);
	r.acc = u->acc_s + 16u * uint32_t((m >> 8) + lane);
	r.col = u->acc_s + 16u * uint32_t(tid);
	r.cstep = 16 * u->rows;
	r.segs = u->segs;
	r.two = u->two;
	r.s0 = r.s1 = 0.0f;
	if (tid < r.ncol) {  // (before the barrier behind which the unit may be refilled)
		r.s0 = ps_ldsf(u->scale_s + 4u * tid);
		if (r.two) r.s1 = ps_ldsf(u->scale_s + 4u * (r.ncol + tid));
	}
	return r;
}
// the segments' digit sums of a column added (exact) and joined
__device__ __forceinline__ float ps_column(const PsRun &r, uint32_t p) {
	int4 s = make_int4(0, 0, 0, 0);
#pragma unroll 4
	for (int i = 0; i < r.segs; i++, p += r.cstep) {
		const uint4 v = ps_lds128(p);
		s.x += int(v.x);
		s.y += int(v.y);
		s.z += int(v.z);
		s.w += int(v.w);
	}
	return ps_join(s);
}
// One unit's product: dst[c] = column sum * scale, or (up and gate) GeLU(gate) * up. Called by the whole CTA behind the
// barrier that ends the prologue (the digits' writers have fenced). Warp 4 t issues tile
// t's MMAs into its own 16 TMEM columns (one accumulator per issuing warp), warps 4 t .. 4 t + 3 read them back, thread c
// publishes column c. One store instruction per 32 columns: scattered over the warps, 16 bytes each, the words of a line that 148
// CTAs poll take 450 clk longer to arrive. pm: parity of bar_m[t], returned. Behind its barrier nobody reads the unit or the digits any
// more. Measured from the prologue's barrier to the values in registers (1B: 27 MMAs of up and gate, 27 of down, 4 of
// O, 9 of q|k|v): about 430 clk + 38 per MMA of 128 rows, 23 per one of 64; dp4a loops over the same tiles took 2400, 1450,
// 850 and 1000 clk and 400 to 600 more to reduce over the lanes.
__device__ __forceinline__ uint32_t ps_unit(const PsW &w, int where, const PsRun &r, uint64_t *bar_m, uint32_t pm, const float *xscale, float *dst, const GeluLut &lut, uint32_t tab_s, uint64_t hint) {
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, t = warp >> 2;
	if (r.steps) {
		if ((warp & 3) == 0) {
			tc_fence_after();
			const uint64_t step = uint64_t(r.mt * 2);
			const uint32_t id = ps_idesc(r.mt);
			if (tc_elect()) {
#pragma unroll 1
				for (int i = 0; i < r.steps; i++) i8_mma<1>(r.d, r.da + uint64_t(i) * step, r.db + uint64_t(i * (2 * PS_XCH / 16)), id, i > 0 ? 1u : 0u);
				i8_commit<1>(&bar_m[t]);
			}
			__syncwarp();
		}
		ps_wait_bulk(w, where, &bar_m[t], pm);
		pm ^= 1u;
		__syncwarp();
		tc_fence_after();
		const int4 v = ps_tmem_ld4(r.taddr);
		if (4 * lane < r.mt) asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(r.acc), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
		tc_fence_before();
	}
	__syncthreads();
	if (tid < r.ncol) {
		const float xs = *xscale;
		float y = (ps_column(r, r.col) * xs) * r.s0;
		if (r.two) y = ps_gelu(lut, (ps_column(r, r.col + 16u * r.ncol) * xs) * r.s1, tab_s, hint) * y;
		if (dst) ps_st(dst + tid, y);
	}
	return pm;
}

// A CTA's unit is one contiguous block of the re-tiled copy: one bulk copy. Called by one lane.
// Piece `i` of a unit, `size` bytes each; the first one announces all of the unit's bytes to its barrier. Called by one lane.
__device__ __forceinline__ void ps_issue_piece(uint8_t *dst, const int8_t *src, uint32_t bytes, uint32_t size, int i, uint64_t *bar, uint64_t hint, const int *abort_flag) {
	if (*(volatile const int *)abort_flag) return;
	const uint32_t at = uint32_t(i) * size;
	if (i == 0) ps_mbar_expect(bar, bytes);
	if (at < bytes) ps_bulk(dst + at, src + at, min(size, bytes - at), bar, hint);
}
__device__ __noinline__ void ps_issue(uint8_t *dst, const int8_t *src, uint32_t bytes, uint64_t *bar, uint64_t pol, const int *abort_flag) {
	if (*(volatile const int *)abort_flag) return;  // a CTA that gave up starts no new copies
	// (no proxy fence: the region was only READ through the generic proxy, and those loads have completed —
	// their values were consumed before the readers signalled that the tile is free)
	ps_mbar_expect(bar, bytes);
	ps_bulk(dst, src, bytes, bar, pol);
}

// Re-tile `ntiles_mat` column tiles x ph.nsplit K-splits of a row-major int8 matrix [K][N] into unit order: unit (split,
// tile0 + t) is a block at dst + (split * ntiles + tile0 + t) * bytes in the layout described at PsPhase, whose rows row0.. hold this
// matrix; the columns' scales follow the weights. One thread per 4 columns x 16 k.
__device__ __forceinline__ uint4 ps_piece(const int8_t *src, size_t N, size_t row0, size_t col0) {  // 4 x 4: word c = column col0 + c
	const uint32_t r0 = *reinterpret_cast<const uint32_t *>(src + row0 * N + col0);
	const uint32_t r1 = *reinterpret_cast<const uint32_t *>(src + (row0 + 1) * N + col0);
	const uint32_t r2 = *reinterpret_cast<const uint32_t *>(src + (row0 + 2) * N + col0);
	const uint32_t r3 = *reinterpret_cast<const uint32_t *>(src + (row0 + 3) * N + col0);
	const uint32_t t0 = __byte_perm(r0, r1, 0x5140), t1 = __byte_perm(r2, r3, 0x5140);
	const uint32_t t2 = __byte_perm(r0, r1, 0x7362), t3 = __byte_perm(r2, r3, 0x7362);
	return make_uint4(__byte_perm(t0, t1, 0x5410), __byte_perm(t0, t1, 0x7632), __byte_perm(t2, t3, 0x5410), __byte_perm(t2, t3, 0x7632));
}
__global__ void retile_units_kernel(int8_t *dst, const int8_t *src, const float *scales, int N, PsPhase ph, int tile0, int ntiles_mat, int row0) {
	const int gcols = ntiles_mat * ph.ncol / 4, uch = ph.nq / 4, sch = ph.seg_q / 4;  // column groups; 16-k chunks of a unit, of a segment
	const size_t total = size_t(gcols) * uch * ph.nsplit;
	for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x) {
		const int g = int(i % gcols), kc = int(i / gcols);
		const int t = g * 4 / ph.ncol, c = g * 4 - t * ph.ncol, split = kc / uch, ku = kc - split * uch, seg = ku / sch, ch = ku - seg * sch;
		uint4 p[4];
#pragma unroll
		for (int j = 0; j < 4; j++) p[j] = ps_piece(src, size_t(N), size_t(kc) * 16 + 4 * j, size_t(g) * 4);
		uint4 *o = reinterpret_cast<uint4 *>(dst + size_t(split * ph.ntiles + tile0 + t) * ph.bytes + ps_unit_offset(ph, row0 + c, seg, ch));
		o[0] = make_uint4(p[0].x, p[1].x, p[2].x, p[3].x);
		o[1] = make_uint4(p[0].y, p[1].y, p[2].y, p[3].y);
		o[2] = make_uint4(p[0].z, p[1].z, p[2].z, p[3].z);
		o[3] = make_uint4(p[0].w, p[1].w, p[2].w, p[3].w);
	}
	if (!scales) return;
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N * ph.nsplit; i += gridDim.x * blockDim.x) {
		const int split = i / N, n = i - split * N, t = n / ph.ncol, c = n - t * ph.ncol;
		reinterpret_cast<float *>(dst + size_t(split * ph.ntiles + tile0 + t) * ph.bytes + size_t(ph.rows) * ph.nq * 4)[row0 + c] = scales[n];
	}
}

// ------------------------------------------------------------------ prologues
// 1 / sqrt(sumsq / dim + eps): the hardware estimate refined by one Newton step, which is how the
// reference's build evaluates it (rsqrtss + one step under -ffast-math, reference ops.hpp:153)
__device__ __forceinline__ float ps_inv_rms(float sumsq, float inv_dim) {
	const float v = fmaf(sumsq, inv_dim, RMS_EPS);
	const float r = rsqrtf(v);
	return r * fmaf(-0.5f * v, r * r, 1.5f);
}
// If part: t[d] = sum_s part[s][d] (scaled partial sums, polled until complete; threads past D/4 poll
// the presence words);  h += rmsnorm(t; w_post). Then y = rmsnorm(h; w_pre), quantised with *s_xscale = 2^(e - 30).
// Every CTA computes the same bits. D <= 4 * PS_THREADS. Thread t owns elements 4t..4t+3, which are quad t. bred: 3 * PS_NW
// floats, 16-byte aligned.
__device__ __forceinline__ void ps_resnorm(const PsW w, int where, int D, float *h, const PsUnit *u, float *bred, float *s_xscale,
                                        const float *part, int nsplit, const float *pres, int npres, const float *w_post,
                                        const float *w_pre, uint64_t keep, float *x_out) {
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	// the norm weights are L2-resident (evict-last): requested together with the first poll loads
	float4 wpost = make_float4(0.f, 0.f, 0.f, 0.f), wpre = wpost;
	if (4 * tid < D) {
		if (part) wpost = ps_ldk4(w_post + 4 * tid, keep);
		wpre = ps_ldk4(w_pre + 4 * tid, keep);
	}
	const uint32_t bred_s = ps_smem(bred);
	const float invD = 1.0f / float(D);
	const bool in = 4 * tid < D;
	const uint32_t xaddr = ps_xaddr(u, tid);
	float4 hv = make_float4(0.f, 0.f, 0.f, 0.f);
	if (in) hv = *reinterpret_cast<const float4 *>(h + 4 * tid);
	if (part) {
		float4 tv = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
		for (int s0 = 0; s0 < nsplit; s0 += 2) {
			float4 p0, p1;
			int spins = 0;
			long long t0 = 0;
			bool ok;
			do {
				p0 = p1 = make_float4(0.f, 0.f, 0.f, 0.f);
				if (in) {
					p0 = ps_ld4(part + size_t(s0) * D + 4 * tid);
					if (s0 + 1 < nsplit) p1 = ps_ld4(part + size_t(s0 + 1) * D + 4 * tid);
				}
				ok = ps_ok(p0) && ps_ok(p1);
				if (s0 == 0 && !in && tid - D / 4 < npres) ok = ps_ok(ps_ld1(pres + (tid - D / 4)));
			} while (!ok && ps_retry(w, where, spins, t0));
			tv.x += p0.x + p1.x;  // splits in ascending order (p1 is an exact zero when absent)
			tv.y += p0.y + p1.y;
			tv.z += p0.z + p1.z;
			tv.w += p0.w + p1.w;
		}
		float ss = fmaf(tv.x, tv.x, fmaf(tv.y, tv.y, fmaf(tv.z, tv.z, tv.w * tv.w)));
		ss = warp_sum(ss);
		if (lane == 0) ps_stsf(bred_s + 4u * warp, ss);
		__syncthreads();
		const float r1 = ps_inv_rms(ps_sum12(bred_s), invD);
		hv.x = hv.x + (tv.x * r1) * (wpost.x + 1.0f);
		hv.y = hv.y + (tv.y * r1) * (wpost.y + 1.0f);
		hv.z = hv.z + (tv.z * r1) * (wpost.z + 1.0f);
		hv.w = hv.w + (tv.w * r1) * (wpost.w + 1.0f);
		if (in) *reinterpret_cast<float4 *>(h + 4 * tid) = hv;
	}
	const float4 g = make_float4(wpre.x + 1.0f, wpre.y + 1.0f, wpre.z + 1.0f, wpre.w + 1.0f);
	float ss2 = fmaf(hv.x, hv.x, fmaf(hv.y, hv.y, fmaf(hv.z, hv.z, hv.w * hv.w)));
	float mx = fmaxf(fmaxf(fabsf(hv.x * g.x), fabsf(hv.y * g.y)), fmaxf(fabsf(hv.z * g.z), fabsf(hv.w * g.w)));
	mx = ps_warp_max(mx);
	ss2 = warp_sum(ss2);
	if (lane == 0) {
		ps_stsf(bred_s + 4u * (PS_NW + warp), ss2);
		ps_stsf(bred_s + 4u * (2 * PS_NW + warp), mx);
	}
	__syncthreads();
	const float r2 = ps_inv_rms(ps_sum12(bred_s + 4u * PS_NW), invD), M = r2 * ps_max12(bred_s + 8u * PS_NW);
	if (in) {
		float4 y;
		y.x = (hv.x * r2) * g.x;
		y.y = (hv.y * r2) * g.y;
		y.z = (hv.z * r2) * g.z;
		y.w = (hv.w * r2) * g.w;
		ps_quantise(y, ps_qmul(M), xaddr);
		ps_fence_async();
		if (x_out) *reinterpret_cast<float4 *>(x_out + 4 * tid) = y;
	}
	if (tid == 0) *s_xscale = ps_qscale(M);
	__syncthreads();
}

// one warp: x[0..256) (dims 4 lane.. and 128 + 4 lane..) -> rmsnorm, RoPE, * scale
struct PsRope {
	float4 c0, c1, s0, s1;
};
__device__ __forceinline__ void ps_norm_rope(const float4 &lo4, const float4 &hi4, const float4 &w0_, const float4 &w1_, const PsRope &r, float scale, float4 &ylo4, float4 &yhi4) {
	const float lo[4] = {lo4.x, lo4.y, lo4.z, lo4.w}, hi[4] = {hi4.x, hi4.y, hi4.z, hi4.w};
	const float w0[4] = {w0_.x, w0_.y, w0_.z, w0_.w}, w1[4] = {w1_.x, w1_.y, w1_.z, w1_.w};
	const float c0[4] = {r.c0.x, r.c0.y, r.c0.z, r.c0.w}, c1[4] = {r.c1.x, r.c1.y, r.c1.z, r.c1.w};
	const float s0[4] = {r.s0.x, r.s0.y, r.s0.z, r.s0.w}, s1[4] = {r.s1.x, r.s1.y, r.s1.z, r.s1.w};
	float ss = 0.0f;
#pragma unroll
	for (int i = 0; i < 4; i++) {
		ss = fmaf(lo[i], lo[i], ss);
		ss = fmaf(hi[i], hi[i], ss);
	}
	ss = warp_sum(ss);
	const float rr = inv_rms(ss, AT_HD);
	float ylo[4], yhi[4];
#pragma unroll
	for (int i = 0; i < 4; i++) {
		const float p = (lo[i] * rr) * (w0[i] + 1.0f);
		const float q = (hi[i] * rr) * (w1[i] + 1.0f);
		// y = cos * x + rotate_half(x) * sin, rotate_half = [-x_hi, x_lo] (reference decode.hpp:203-211)
		ylo[i] = fmaf(-1.0f * q, s0[i], c0[i] * p) * scale;
		yhi[i] = fmaf(p, s1[i], c1[i] * q) * scale;
	}
	ylo4 = make_float4(ylo[0], ylo[1], ylo[2], ylo[3]);
	yhi4 = make_float4(yhi[0], yhi[1], yhi[2], yhi[3]);
}

// Phase C prologue: merge the attention partials of `hp` heads starting at head h0 over `nch` chunks
// into the normalised output (reference ops.hpp:316-357 keeps it normalised per step; the split form
// divides once), quantise it.
__device__ __forceinline__ void ps_attn_merge(const PsW w, int where, const float *att_ll, int h0, int hp, int nch, float *scr, const PsUnit *u, float *bred,
                                              float *s_xscale) {
	const int tid = threadIdx.x;
	// thread = (chunk group cg, float4 column it of the hp * 64); hp is 1, 2 or 4
	const int sh = 6 + (hp >> 1), items = 1 << sh;
	const int ncg = hp == 1 ? PS_THREADS / 64 : (hp == 2 ? PS_THREADS / 128 : PS_THREADS / 256);
	const int cg = tid >> sh, it = tid & (items - 1);
	const int hl = it >> 6, j = it & 63;
	const uint32_t xaddr = ps_xaddr(u, it);
	float m = -INFINITY, l = 0.0f;
	float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
	if (cg < ncg) {
		// PB chunks are requested together: one after the other a hand-off of nine chunks took three dependent round trips
		constexpr int PB = 4;
#pragma unroll 1
		for (int cb = cg; cb < nch; cb += PB * ncg) {
			float4 ov[PB];
			float2 ml[PB];
			int spins = 0;
			long long t0 = 0;
			bool ok;
			do {
				ok = true;
#pragma unroll
				for (int i = 0; i < PB; i++) {
					const int ch = cb + i * ncg;
					ml[i] = make_float2(-INFINITY, 0.0f);
					ov[i] = make_float4(0.f, 0.f, 0.f, 0.f);
					if (ch < nch) {
						const float *r0 = att_ll + (size_t(h0 + hl) * PS_MAX_CH + ch) * PS_ATT_ROW;
						ov[i] = ps_ld4(r0 + 4 * j);
						ml[i] = ps_ld2(r0 + AT_HD);
					}
				}
#pragma unroll
				for (int i = 0; i < PB; i++) ok = ok && ps_ok(ov[i]) && ps_ok(ml[i]);
			} while (!ok && ps_retry(w, where, spins, t0));
			float mn = m;
#pragma unroll
			for (int i = 0; i < PB; i++) mn = fmaxf(mn, ml[i].x);
			if (mn == -INFINITY) continue;  // nothing but empty chunks so far
			const float ea = expf(m - mn);
			l *= ea;
			o.x *= ea;
			o.y *= ea;
			o.z *= ea;
			o.w *= ea;
#pragma unroll
			for (int i = 0; i < PB; i++) {
				const float eb = expf(ml[i].x - mn);
				l = fmaf(ml[i].y, eb, l);
				o.x = fmaf(ov[i].x, eb, o.x);
				o.y = fmaf(ov[i].y, eb, o.y);
				o.z = fmaf(ov[i].z, eb, o.z);
				o.w = fmaf(ov[i].w, eb, o.w);
			}
			m = mn;
		}
	}
	__syncthreads();  // (the attention of this CTA has left the scratch)
	if (cg < ncg) {
		float *s = scr + (size_t(cg) * items + it) * 8;
		*reinterpret_cast<float4 *>(s) = o;
		*reinterpret_cast<float2 *>(s + 4) = make_float2(m, l);
	}
	__syncthreads();
	float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
	float mx = 0.0f;
	if (tid < items) {
		constexpr int NG = PS_THREADS / 64;
		float mg[NG], M = -INFINITY, L = 0.0f;
#pragma unroll
		for (int g = 0; g < NG; g++) {
			mg[g] = g < ncg ? scr[(size_t(g) * items + tid) * 8 + 4] : -INFINITY;
			M = fmaxf(M, mg[g]);
		}
#pragma unroll
		for (int g = 0; g < NG; g++) {
			if (g >= ncg) break;
			const float *s = scr + (size_t(g) * items + tid) * 8;
			const float e = expf(mg[g] - M);
			const float4 ov = *reinterpret_cast<const float4 *>(s);
			L = fmaf(s[5], e, L);
			y.x = fmaf(ov.x, e, y.x);
			y.y = fmaf(ov.y, e, y.y);
			y.z = fmaf(ov.z, e, y.z);
			y.w = fmaf(ov.w, e, y.w);
		}
		const float inv = 1.0f / L;
		y.x *= inv;
		y.y *= inv;
		y.z *= inv;
		y.w *= inv;
		mx = fmaxf(fmaxf(fabsf(y.x), fabsf(y.y)), fmaxf(fabsf(y.z), fabsf(y.w)));
	}
	const float M = ps_block_max(mx, bred);
	if (tid < items) {
		ps_quantise(y, ps_qmul(M), xaddr);
		ps_fence_async();
	}
	if (tid == 0) *s_xscale = ps_qscale(M);
	__syncthreads();
}

// Phase E prologue: this CTA's rows of the activation vector (nq quads from act), polled until
// complete, quantised. nq <= PS_ACT * PS_THREADS.
__device__ __forceinline__ void ps_act_quant(const PsW w, int where, const float *act, int nq, const PsUnit *u, float *bred, float *s_xscale) {
	const int tid = threadIdx.x;
	float4 v[PS_ACT];
	int spins = 0;
	long long t0 = 0;
	bool ok;
	do {
		ok = true;
#pragma unroll
		for (int q = 0; q < PS_ACT; q++) {
			const int i = q * PS_THREADS + tid;
			v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
			if (i < nq) v[q] = ps_ld4(act + 4 * i);
			ok = ok && ps_ok(v[q]);
		}
	} while (!ok && ps_retry(w, where, spins, t0));
	float mx = 0.0f;
#pragma unroll
	for (int q = 0; q < PS_ACT; q++) mx = fmaxf(mx, fmaxf(fmaxf(fabsf(v[q].x), fabsf(v[q].y)), fmaxf(fabsf(v[q].z), fabsf(v[q].w))));
	const float M = ps_block_max(mx, bred);
	const float qs = ps_qmul(M);
#pragma unroll
	for (int q = 0; q < PS_ACT; q++) {
		const int i = q * PS_THREADS + tid;
		if (i < nq) ps_quantise(v[q], qs, ps_xaddr(u, i));
	}
	if (tid == 0) *s_xscale = ps_qscale(M);
	ps_fence_async();
	__syncthreads();
}

// Phase B of one attention CTA = (head hh, cache slots j0 .. j1): q|k|v of this token from the hand-off
// vector (polled), q/k norm + RoPE, append of the new row (head 0's CTA of the chunk that holds `slot`),
// running-max softmax over the chunk (warp -> slots j0 + warp, + 12, ...; lane owns dims 4 lane.. and
// 128 + 4 lane..), merge of the 12 warps, (o[256], m, l) published to prow. att: 16 KB of scratch,
// wml: 2 * PS_NW floats. Every warp norms and rotates q itself, the one that owns the new row k too: one barrier less, and
// no values through shared memory. Reference: ops.hpp:224-370 (attention_decode), decode.hpp:203-211 (RoPE).
__device__ __forceinline__ void ps_attention(const PsW w, int where, float *kcache, float *vcache, const float *rmsq, const float *rmsk,
                                          const float *cosr, const float *sinr, const float *qkv_ll, int QD, int hh, float *prow, int j0,
                                          int j1, int slot, float *att, float *wml, uint64_t keep) {
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	float *wo = att, *qraw = att + PS_NW * AT_HD;
	float *wm = wml, *wl = wml + PS_NW;
	// The cache rows do not depend on this token's q|k|v: a warp's first two rows are requested before
	// the poll (the new token's own row comes from shared memory later).
	float4 kv[2][4];
	auto load_keys = [&](int jb) {
#pragma unroll
		for (int u = 0; u < 2; u++) {
			const int j = jb + PS_NW * u;
#pragma unroll
			for (int i = 0; i < 4; i++) kv[u][i] = make_float4(0.f, 0.f, 0.f, 0.f);
			if (j < j1 && j != slot) {
				const float *kr = kcache + size_t(j) * AT_HD, *vr = vcache + size_t(j) * AT_HD;
				kv[u][0] = __ldcg(reinterpret_cast<const float4 *>(kr + 4 * lane));
				kv[u][1] = __ldcg(reinterpret_cast<const float4 *>(kr + 128 + 4 * lane));
				kv[u][2] = __ldcg(reinterpret_cast<const float4 *>(vr + 4 * lane));
				kv[u][3] = __ldcg(reinterpret_cast<const float4 *>(vr + 128 + 4 * lane));
			}
		}
	};
	load_keys(j0 + warp);
	const bool own = slot >= j0 && slot < j1 && (slot - j0) % PS_NW == warp;
	PsRope rr;
	rr.c0 = ps_ldk4(cosr + 4 * lane, keep);
	rr.c1 = ps_ldk4(cosr + 128 + 4 * lane, keep);
	rr.s0 = ps_ldk4(sinr + 4 * lane, keep);
	rr.s1 = ps_ldk4(sinr + 128 + 4 * lane, keep);
	const float4 wq0 = ps_ldk4(rmsq + 4 * lane, keep), wq1 = ps_ldk4(rmsq + 128 + 4 * lane, keep);
	float4 wk0 = wq0, wk1 = wq1;
	if (own) {
		wk0 = ps_ldk4(rmsk + 4 * lane, keep);
		wk1 = ps_ldk4(rmsk + 128 + 4 * lane, keep);
	}
	if (tid < 3 * (AT_HD / 4)) {
		const float *src = qkv_ll + (tid < AT_HD / 4 ? hh * AT_HD + 4 * tid : QD + 4 * (tid - AT_HD / 4));
		float4 v;
		int spins = 0;
		long long t0 = 0;
		do {
			v = ps_ld4(src);
		} while (!ps_ok(v) && ps_retry(w, where, spins, t0));
		*reinterpret_cast<float4 *>(qraw + 4 * tid) = v;
	}
	__syncthreads();
	const float4 *q4 = reinterpret_cast<const float4 *>(qraw);
	float4 q0, q1, k0, k1;
	// the reference scales q by 1/sqrt(256) before the dot products (ops.hpp:262,283); k is normed in place
	ps_norm_rope(q4[lane], q4[32 + lane], wq0, wq1, rr, 0.0625f, q0, q1);
	if (own) ps_norm_rope(q4[64 + lane], q4[96 + lane], wk0, wk1, rr, 1.0f, k0, k1);
	float4 o0 = make_float4(0.f, 0.f, 0.f, 0.f), o1 = make_float4(0.f, 0.f, 0.f, 0.f);
	float m = -INFINITY, lsum = 0.0f;
#pragma unroll 1
	for (int jb = j0 + warp; jb < j1; jb += 2 * PS_NW) {
#pragma unroll
		for (int u = 0; u < 2; u++)
			if (own && jb + PS_NW * u == slot) {  // the new row: not in the cache yet for the other heads' CTAs
				kv[u][0] = k0;
				kv[u][1] = k1;
				kv[u][2] = q4[128 + lane];
				kv[u][3] = q4[160 + lane];
				if (hh == 0) {
					float4 *kr = reinterpret_cast<float4 *>(kcache + size_t(slot) * AT_HD), *vr = reinterpret_cast<float4 *>(vcache + size_t(slot) * AT_HD);
					kr[lane] = k0;
					kr[32 + lane] = k1;
					vr[lane] = kv[u][2];
					vr[32 + lane] = kv[u][3];
				}
			}
		// two rows at a time: their sums over the lanes overlap
		float t[2];
#pragma unroll
		for (int u = 0; u < 2; u++) {
			t[u] = q0.x * kv[u][0].x;
			t[u] = fmaf(q0.y, kv[u][0].y, t[u]);
			t[u] = fmaf(q0.z, kv[u][0].z, t[u]);
			t[u] = fmaf(q0.w, kv[u][0].w, t[u]);
			t[u] = fmaf(q1.x, kv[u][1].x, t[u]);
			t[u] = fmaf(q1.y, kv[u][1].y, t[u]);
			t[u] = fmaf(q1.z, kv[u][1].z, t[u]);
			t[u] = fmaf(q1.w, kv[u][1].w, t[u]);
		}
#pragma unroll
		for (int of = 16; of > 0; of >>= 1) {
			t[0] += __shfl_xor_sync(0xffffffffu, t[0], of);
			t[1] += __shfl_xor_sync(0xffffffffu, t[1], of);
		}
		if (jb + PS_NW >= j1) t[1] = -INFINITY;  // (its values are zeros)
		const float mn = fmaxf(m, fmaxf(t[0], t[1]));
		const float corr = expf(m - mn), p0 = expf(t[0] - mn), p1 = expf(t[1] - mn);
		lsum = fmaf(lsum, corr, p0) + p1;
		o0.x = fmaf(p1, kv[1][2].x, fmaf(p0, kv[0][2].x, o0.x * corr));
		o0.y = fmaf(p1, kv[1][2].y, fmaf(p0, kv[0][2].y, o0.y * corr));
		o0.z = fmaf(p1, kv[1][2].z, fmaf(p0, kv[0][2].z, o0.z * corr));
		o0.w = fmaf(p1, kv[1][2].w, fmaf(p0, kv[0][2].w, o0.w * corr));
		o1.x = fmaf(p1, kv[1][3].x, fmaf(p0, kv[0][3].x, o1.x * corr));
		o1.y = fmaf(p1, kv[1][3].y, fmaf(p0, kv[0][3].y, o1.y * corr));
		o1.z = fmaf(p1, kv[1][3].z, fmaf(p0, kv[0][3].z, o1.z * corr));
		o1.w = fmaf(p1, kv[1][3].w, fmaf(p0, kv[0][3].w, o1.w * corr));
		m = mn;
		if (jb + 2 * PS_NW < j1) load_keys(jb + 2 * PS_NW);
	}
	if (lane == 0) {
		wm[warp] = m;
		wl[warp] = lsum;
	}
	*reinterpret_cast<float4 *>(wo + warp * AT_HD + 4 * lane) = o0;
	*reinterpret_cast<float4 *>(wo + warp * AT_HD + 128 + 4 * lane) = o1;
	__syncthreads();
	// merge: lane i of every warp holds warp i's maximum and weight (the caller's next use of the scratch is behind a barrier)
	if (warp <= AT_HD / 32) {
		const float mi = lane < PS_NW ? wm[lane] : -INFINITY;
		const float M = warp_max(mi);
		const float e = mi == -INFINITY ? 0.0f : expf(mi - M);
		if (warp < AT_HD / 32) {
			float O = 0.0f;
#pragma unroll
			for (int i = 0; i < PS_NW; i++) O = fmaf(wo[i * AT_HD + tid], __shfl_sync(0xffffffffu, e, i), O);
			ps_st(prow + tid, O);
		} else {
			const float li = lane < PS_NW ? wl[lane] : 0.0f;
			float Ls = 0.0f;
#pragma unroll
			for (int i = 0; i < PS_NW; i++) Ls = fmaf(__shfl_sync(0xffffffffu, li, i), __shfl_sync(0xffffffffu, e, i), Ls);
			if (lane < 2) ps_st(prow + AT_HD + lane, lane == 0 ? M : Ls);
		}
	}
}

// lm_head of one token: logits[v] = lm_scale[v] * sum_k x[k] W[k,v]; this CTA takes tiles cta, cta + G, ... of 128 columns; a
// tile arrives as lm_nchunk ring stages in `ring`. Warp PS_NW - 1 copies, warp 8 multiplies into one of two accumulators, warps
// 0 to 3 take 32 columns each. Returns this lane's best (temperature-scaled) logit and the ring's barrier parities.
// pre: ring stages the caller has already requested (those that lie inside the up/gate region, which is
// idle from the last layer's up/gate product on). acc_n: tiles of this CTA so far.
// HBM bounds it. With dp4a products on all 12 warps a stage took about as long to multiply as to arrive, and 302 MB took 57.6 us;
// a copy into the same rings that multiplies nothing takes 49.
struct PsLmOut {
	float best;
	int best_i;
	uint32_t plm, pemp;
};
__device__ __noinline__ PsLmOut ps_lm_head(const PsArgs &a, const PsW pw, uint8_t *ring, uint32_t smem_s, float xs, uint32_t tmem, uint64_t *bar_lm,
                                           uint64_t *emp_lm, uint64_t *acc_full, uint64_t *acc_free, uint32_t plm, uint32_t pemp, uint32_t acc_n,
                                           uint64_t pol, uint64_t keep, int pre) {
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int cta = blockIdx.x, G = gridDim.x, where = (a.L << 4) | 6;
	__builtin_assume(__isShared(ring));
	const int nst = a.lm_stages, nchunk = a.lm_nchunk, my_tiles = (a.lm_ntiles - cta + G - 1) / G, total = my_tiles * nchunk;
	const uint32_t sbytes = uint32_t(a.lm_stage_bytes);
	PsLmOut o{-INFINITY, -1, plm, pemp};
	if (warp == PS_NW - 1) {
		int t = cta, c = pre, stg = pre;  // (pre <= nchunk)
		if (c == nchunk) {
			c = 0;
			t += G;
		}
		if (stg == nst) stg = 0;
#pragma unroll 1
		for (int q = pre; q < total; q++) {
			if (q >= nst) {
				ps_wait_bulk(pw, where, &emp_lm[stg], (pemp >> stg) & 1u);
				pemp ^= 1u << stg;
			}
			__syncwarp();
			if (tc_elect()) ps_issue(ring + size_t(stg) * sbytes, a.lm_tiled + (size_t(t) * nchunk + c) * sbytes, sbytes, &bar_lm[stg], pol, pw.s_abort);
			__syncwarp();
			if (++stg == nst) stg = 0;
			if (++c == nchunk) {
				c = 0;
				t += G;
			}
		}
	} else if (warp == 8) {
		const uint32_t id = ps_idesc(128);
		const uint64_t db0 = ps_desc(smem_s + uint32_t(a.lm.off_x), PS_XCH, a.lm.x_sbo);
		int stg = 0, c = 0;
#pragma unroll 1
		for (int q = 0; q < total; q++) {
			const uint32_t b = acc_n & 1u;
			if (c == 0) ps_wait_bulk(pw, where, &acc_free[b], ((acc_n >> 1) & 1u) ^ 1u);  // (the first use of a fresh barrier passes)
			ps_wait_bulk(pw, where, &bar_lm[stg], (plm >> stg) & 1u);
			plm ^= 1u << stg;
			__syncwarp();
			tc_fence_after();
			const uint64_t da = ps_desc(ps_smem(ring) + uint32_t(stg) * sbytes, 128 * 16, 128), db = db0 + uint64_t(c * a.lm_steps * (2 * PS_XCH / 16));
			if (tc_elect()) {
#pragma unroll 1
				for (int i = 0; i < a.lm_steps; i++) i8_mma<1>(tmem + 16u * b, da + uint64_t(i * 256), db + uint64_t(i * (2 * PS_XCH / 16)), id, (c | i) ? 1u : 0u);
				i8_commit<1>(&emp_lm[stg]);
				if (c == nchunk - 1) i8_commit<1>(&acc_full[b]);
			}
			__syncwarp();
			if (++stg == nst) stg = 0;
			if (++c == nchunk) {
				c = 0;
				acc_n++;
			}
		}
	} else if (warp < 4) {
#pragma unroll 1
		for (int t = cta; t < a.lm_ntiles; t += G, acc_n++) {
			const int v = t * 128 + warp * 32 + lane;
			const float sc = ps_ldk(a.lm_scale + v, keep);
			const uint32_t b = acc_n & 1u;
			ps_wait_bulk(pw, where, &acc_full[b], (acc_n >> 1) & 1u);
			__syncwarp();
			tc_fence_after();
			const int4 s = ps_tmem_ld4(tmem + (uint32_t(warp * 32) << 16) + 16u * b);
			tc_fence_before();
			__syncwarp();
			if (lane == 0) ps_mbar_arrive(&acc_free[b]);
			const float lg = (ps_join(s) * xs) * sc;
			__stcg(a.logits + v, lg);
			const float z = (a.sampler == 2) ? lg / a.temp : lg;
			if (z > o.best) {  // tiles ascend, so the first maximum keeps the lowest index
				o.best = z;
				o.best_i = v;
			}
		}
	}
	// every slot's barriers have completed once per use
#pragma unroll 1
	for (int s = 0; s < nst && s < total; s++)
		if ((((total - s + nst - 1) / nst) & 1) != 0) {
			o.plm ^= 1u << s;
			o.pemp ^= 1u << s;
		}
	return o;
}

// Sampler of one token (0: none, 1: argmax, 2: min-p) over the logits row; `best`, `best_i` are this lane's
// candidates from the lm_head. Returns the sampled token (every thread) and the grid-barrier count.
struct PsSampOut {
	int tok;
	unsigned epoch;
};
__device__ __noinline__ PsSampOut ps_sampler(const PsArgs &a, const PsW pw, float best, int best_i, unsigned epoch, int n_logged, float *wm,
                                             int *s_cdf, float *s_f, int *s_i, float *bred, float *cbuf) {
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int cta = blockIdx.x, G = gridDim.x, L = a.L;
	// these are shared-memory pointers: tell the compiler, or every access through them is a generic load
	__builtin_assume(__isShared(wm));
	__builtin_assume(__isShared(s_cdf));
	__builtin_assume(__isShared(s_f));
	__builtin_assume(__isShared(s_i));
	__builtin_assume(__isShared(bred));
	__builtin_assume(__isShared(cbuf));
const int wh = (L << 4) | 7;
int next_tok = 0;
if (a.sampler == 0) {
	ps_grid_sync(pw, wh, a.bar, a.bar_base + ++epoch * G);  // logits complete
} else {
	// CTA-local (max, argmax): value descending, index ascending; index -1 never beats a real one
	auto better = [](float v1, int i1, float v2, int i2) {
		if (v1 > v2) return true;
		if (v1 < v2) return false;
		if (i2 < 0) return i1 >= 0;
		if (i1 < 0) return false;
		return i1 < i2;
	};
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) {
		float ov = __shfl_xor_sync(0xffffffffu, best, o);
		int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
		if (better(ov, oi, best, best_i)) {
			best = ov;
			best_i = oi;
		}
	}
	if (lane == 0) {
		wm[warp] = best;
		s_cdf[warp] = best_i;
	}
	__syncthreads();
	if (tid == 0) {
		for (int i = 1; i < PS_NW; i++)
			if (better(wm[i], s_cdf[i], best, best_i)) {
				best = wm[i];
				best_i = s_cdf[i];
			}
		__stcg(a.samp_f + cta, best);
		__stcg(a.samp_i + cta, best_i);
	}
	ps_grid_sync(pw, wh, a.bar, a.bar_base + ++epoch * G);
	// every CTA reduces the per-CTA results the same way (warp 0)
	if (warp == 0) {
		float gmax = -INFINITY;
		int gidx = -1;
#pragma unroll 1
		for (int cb = lane; cb < G; cb += 32 * 5) {  // (five loads of each in flight)
			float v[5];
			int ix[5];
#pragma unroll
			for (int q = 0; q < 5; q++) {
				const int c = cb + 32 * q;
				v[q] = c < G ? __ldcg(a.samp_f + c) : -INFINITY;
				ix[q] = c < G ? __ldcg(a.samp_i + c) : -1;
			}
#pragma unroll
			for (int q = 0; q < 5; q++)
				if (better(v[q], ix[q], gmax, gidx)) {
					gmax = v[q];
					gidx = ix[q];
				}
		}
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) {
			float ov = __shfl_xor_sync(0xffffffffu, gmax, o);
			int oi = __shfl_xor_sync(0xffffffffu, gidx, o);
			if (better(ov, oi, gmax, gidx)) {
				gmax = ov;
				gidx = oi;
			}
		}
		if (lane == 0) {
			s_f[4] = gmax;
			s_i[0] = gidx;
		}
	}
	__syncthreads();
	const float gmax = s_f[4];
	const int gidx = s_i[0];
	if (a.sampler == 1) {
		next_tok = gidx;  // ops::argmax_logits (reference ops.hpp:744-760)
	} else {
		// ops::minp_logits (reference ops.hpp:762-859). z = logit / temp; rowmax = gmax;
		// p = exp(z - rowmax); maxp = exp(0) = 1 so cut = minp * 1; denom = sum of p >= cut.
		// The row is worked on in the idle weight ring. (The count is read by every CTA before the barriers
		// behind which CTA 0 raises it.)
		const int rc = __ldcg(a.randf_count);
		const float randf = rc < a.randf_cap ? __ldg(a.randf + rc) : 0.0f;
		next_tok = minp_grid_row<PS_NW>(a.logits, a.probs, a.V, a.minp, a.temp, gmax, randf, a.samp_f, cbuf, bred, s_cdf,
		                             [&] { ps_grid_sync(pw, wh, a.bar, a.bar_base + ++epoch * G); });
		if (cta == 0 && tid == 0) *a.randf_count = rc + 1;
		ps_fence_async();  // (bulk copies refill the ring)
		__syncthreads();
	}
	if (cta == 0 && tid == 0) {
		if (a.tok_log && n_logged < a.log_cap) a.tok_log[n_logged] = next_tok;
		*a.tok = next_tok;
	}
	n_logged++;
}
	return PsSampOut{next_tok, epoch};
}

// Instrumentation of the DBG instantiation only: SM-clock stamps of one CTA along the last token,
// and progress marks of every warp in mapped host memory (for diagnosing a stall).
#define PS_BEACON(x)                                                                               \
	do {                                                                                           \
		if constexpr (DBG) {                                                                       \
			if (a.beacon && lane == 0) *(volatile int *)(a.beacon + cta * 16 + warp) = (lc << 8) | (x); \
		}                                                                                          \
	} while (0)
#define PS_GT(k)                                                                                        \
	do {                                                                                                \
		if constexpr (DBG) {                                                                            \
			if (a.gt && tid == 0 && !more && l == L / 2) {                                              \
				unsigned long long t_;                                                                  \
				asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_));                                  \
				a.gt[cta * 12 + (k)] = (long long)t_;                                                   \
			}                                                                                           \
		}                                                                                               \
	} while (0)
#define PS_GT_WARP(k)                                                                                   \
	do {                                                                                                \
		if constexpr (DBG) {                                                                            \
			if (a.gt && lane == 0 && !more && l == L / 2) {                                             \
				unsigned long long t_;                                                                  \
				asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_));                                  \
				a.gt[cta * 12 + (k)] = (long long)t_;                                                   \
			}                                                                                           \
		}                                                                                               \
	} while (0)
#define PS_STAMP()                                                       \
	do {                                                                 \
		if constexpr (DBG) {                                             \
			if (dbg_on && s_dbg_n < a.dbg_cap) a.dbg[s_dbg_n++] = clock64(); \
		}                                                                \
	} while (0)

// ------------------------------------------------------------------ the kernel's shared memory
// (at namespace scope: a layer's code, which is a function of its own, addresses it without pointers)
extern __shared__ uint8_t ps_dyn[];
__shared__ PsArgs s_args;  // (the arguments, for the functions)
__shared__ uint64_t bar_A, bar_C, bar_D, bar_E, bar_lm[8], emp_lm[8];
__shared__ uint64_t bar_m[PS_TILES], acc_full[2], acc_free[2];  // MMAs of a unit's tile; the lm_head's two accumulators
__shared__ __align__(16) float bred[3 * PS_NW];
__shared__ uint32_t s_tmem;
__shared__ float s_xscale;
__shared__ int s_abort;
__shared__ float s_f[8];
__shared__ int s_i[4];
__shared__ int s_cdf[2 * PS_NW + 8];
__shared__ float wm[2 * PS_NW];  // per-warp (m, l) of the attention merge; also the sampler's per-warp maxima
__shared__ PsLayer s_ly[PS_MAX_LAYERS];
__shared__ PsUnit s_u[5];  // A, C, D, E, lm_head
__shared__ PsSpan s_at[2];  // [is_local]
__shared__ PsCta s_c;
__shared__ PsLive s_t;
__shared__ int s_dbg_n;

#define R_A (smem + a.off_A)
#define R_C (smem + a.off_C)
#define R_D (smem + a.off_D)
#define R_E (smem + a.off_E)
// (recomputed where they are used: a value that lives across the whole token loop costs a register, and the
// registers this kernel cannot have are spilled to local memory, which the small L1 left beside 224 KB of
// shared memory does not hold)
#define h (reinterpret_cast<float *>(smem + a.off_h))
#define att (reinterpret_cast<float *>(smem + a.off_att))  /* wo[12][256] | qraw[768] (q_h, k, v) | qs[256] */
#define smem_s (ps_smem(smem))
#define tmem (s_c.tm)
#define lut_s (smem_s + uint32_t(a.off_lut))
#define pol (s_c.policy_first)
#define keep (s_c.policy_last)

#define hasA ((s_c.has & 1) != 0)
#define hasC ((s_c.has & 2) != 0)
#define hasD ((s_c.has & 4) != 0)
#define hasE ((s_c.has & 8) != 0)

#define lm_pre (cta < a.lm_ntiles ? a.lm_pre : 0)

__device__ __noinline__ void ps_final_norm(const PsW w, int where, int D, float *h_, const PsUnit *u, float *s_x, const float *part, int nsplit,
                                           const float *pres, int npres, const float *w_post, const float *w_pre, uint64_t hint, float *x_out) {
	ps_resnorm(w, where, D, h_, u, bred, s_x, part, nsplit, pres, npres, w_post, w_pre, hint, x_out);
}

// The up/gate and the down unit of a layer are requested in four pieces each, from the layer before on: at the start of phase E
// (the up/gate region is free), A (the down region is free), B, C and D, under the poll that begins there. Requested at once, the
// 24 MB of all CTAs held up the hand-off that they met by 1 to 1.5 us, wherever that was.
#define PS_REFILL_D(layer, i) \
	if (tid == PS_THREADS - 32 && (layer) < L && hasD) ps_issue_piece(R_D, s_c.srcD + size_t(layer) * a.tl_layer, a.Dp.bytes, a.piece_D, i, &bar_D, pol, &s_abort)
#define PS_REFILL_E(layer, i) \
	if (tid == PS_THREADS - 64 && (layer) < L && hasE) ps_issue_piece(R_E, s_c.srcE + size_t(layer) * a.tl_layer, a.E.bytes, a.piece_E, i, &bar_E, pol, &s_abort)
// (No __builtin_assume(__isShared(p)) in what is inlined here: on the address of a shared variable the compiler folds it to
// false and drops the code behind it.)
// One layer. A function of its own, with its phases inlined: a call and its return cost 250 to 350 clk each here (in-kernel
// clocks), and nine calls a layer were a fifth of its time. pm: parity of bar_m, returned.
template <bool DBG> __device__ __noinline__ uint32_t ps_layer(const int l, const int lc, const bool more, uint32_t pm) {
	const PsArgs &a = s_args;
	uint8_t *smem = reinterpret_cast<uint8_t *>((uintptr_t(ps_dyn) + 127) & ~uintptr_t(127));
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int cta = blockIdx.x, G = gridDim.x;
	const int D = a.D, L = a.L;
	const PsW pw{&s_abort, a.err, a.wait_clocks, unsigned(a.poll_ns)};
	const bool dbg_on = DBG && (a.dbg != nullptr) && cta == a.dbg_cta && tid == 0 && !more;
	const PsLayer &ly = s_ly[l];
	const PsSpan &at = s_at[ly.is_local];
	const int nsA = AT_NH * at.nch;  // CTAs that take part in attention
	const uint32_t par = lc & 1;  // parity of the units' barriers: one completion per layer
	const int nl = (l + 1 < L) ? l + 1 : (more ? 0 : -1);  // the layer whose units are fetched next
	float *const llb = a.ll + size_t(lc % 3) * a.ll_stride;
	float *const llprev = a.ll + size_t((lc + 2) % 3) * a.ll_stride;
	PS_BEACON(0x10);
	PS_GT(0);
	// ============================================================ A: QKV
	if (l > 0) {
		PS_REFILL_D(l, 1);
		PS_REFILL_E(l, 0);
	}
	{
		PsRun run;
		if (hasA) run = ps_prepare(pw, (l << 4) | 1, &s_u[0], tmem, &bar_A, par);
		ps_resnorm(pw, (l << 4) | 1, D, h, &s_u[0], bred, &s_xscale, l > 0 ? llprev + a.ll_dn : nullptr, a.E.nsplit, llprev + a.ll_pres,
		           G - a.E.units, l > 0 ? s_ly[l - 1].mlp_post : nullptr, ly.attn_pre, keep, nullptr);
		PS_STAMP();
		PS_GT(1);
		PS_BEACON(0x11);
		if (hasA) {
			PS_STAMP();
			pm = ps_unit(pw, (l << 4) | 1, run, bar_m, pm, &s_xscale, llb + s_u[0].dst, a.lut, lut_s, keep);
			PS_STAMP();
			if (nl >= 0 && tid == PS_THREADS - 32) ps_issue(R_A, s_c.srcA + size_t(nl) * a.tl_layer, a.A.bytes, &bar_A, pol, &s_abort);
		} else {
			PS_STAMP();
			PS_STAMP();
		}
		PS_STAMP();
		PS_GT(2);
		PS_BEACON(0x12);
		// Wipe the arena copy of the NEXT layer. It was last used two layers ago; every CTA has
		// finished with it: this CTA got past the prologue above, which needs the down-projection
		// (or presence) words of ALL CTAs for the previous layer, and a CTA stores those after its
		// last read of anything older. The CTAs that idle through the attention phase wipe; the
		// fence orders the wipe before their own next down-projection / presence store.
		if (cta >= nsA) {
			float4 *other = reinterpret_cast<float4 *>(a.ll + size_t((lc + 1) % 3) * a.ll_stride);
			const int nw = G - nsA, n4 = a.ll_stride / 4, per = (n4 + nw - 1) / nw;
			const float e = __uint_as_float(PS_EMPTY);
#pragma unroll 1
			for (int i = (cta - nsA) * per + tid; i < min(n4, (cta - nsA + 1) * per); i += PS_THREADS)
				__stcg(other + i, make_float4(e, e, e, e));
			__syncthreads();
			if (tid == 0) __threadfence();
		}
		PS_STAMP();
	}
	// ============================================================ B: attention
	if (l > 0) {
		PS_REFILL_D(l, 2);
		PS_REFILL_E(l, 1);
	}
	if (cta < nsA) {
		const int j0 = (cta >> 2) * at.chunk;
		ps_attention(pw, (l << 4) | 2, ly.kcache, ly.vcache, ly.rmsq, ly.rmsk, a.rope[ly.is_local][0] + size_t(at.p) * AT_HD,
		             a.rope[ly.is_local][1] + size_t(at.p) * AT_HD, llb + a.ll_qkv, a.QD, cta & 3,
		             llb + a.ll_att + (size_t(cta & 3) * PS_MAX_CH + (cta >> 2)) * PS_ATT_ROW, j0, min(at.valid, j0 + at.chunk), at.slot, att, wm,
		             keep);
	}
	PS_BEACON(0x24);
	PS_GT(3);
	PS_STAMP();
	// ============================================================ C: O projection
	if (l > 0) {
		PS_REFILL_D(l, 3);
		PS_REFILL_E(l, 2);
	}
	{
		if (hasC) {
			const PsRun run = ps_prepare(pw, (l << 4) | 3, &s_u[1], tmem, &bar_C, par);
			ps_attn_merge(pw, (l << 4) | 3, llb + a.ll_att, s_c.splitC * a.merge_heads, a.merge_heads, at.nch, att, &s_u[1], bred, &s_xscale);
			PS_STAMP();
			PS_GT(4);
			PS_BEACON(0x31);
			PS_STAMP();
			pm = ps_unit(pw, (l << 4) | 3, run, bar_m, pm, &s_xscale, llb + s_u[1].dst, a.lut, lut_s, keep);
			PS_STAMP();
			if (nl >= 0 && tid == PS_THREADS - 32) ps_issue(R_C, s_c.srcC + size_t(nl) * a.tl_layer, a.C.bytes, &bar_C, pol, &s_abort);
		} else {
			PS_STAMP();
			PS_STAMP();
			PS_STAMP();
		}
		PS_STAMP();
		PS_GT(5);
		PS_BEACON(0x32);
	}
	// ============================================================ D: up & gate + GeGLU
	if (l > 0) PS_REFILL_E(l, 3);
	{
		PsRun run;
		if (hasD) run = ps_prepare(pw, (l << 4) | 4, &s_u[2], tmem, &bar_D, par);
		ps_resnorm(pw, (l << 4) | 4, D, h, &s_u[2], bred, &s_xscale, llb + a.ll_op, a.C.nsplit, nullptr, 0, ly.attn_post, ly.mlp_pre, keep, nullptr);
		PS_STAMP();
		PS_GT(6);
		PS_BEACON(0x41);
		PS_STAMP();
		if (hasD) pm = ps_unit(pw, (l << 4) | 4, run, bar_m, pm, &s_xscale, llb + s_u[2].dst, a.lut, lut_s, keep);
		PS_STAMP();
		PS_GT(7);
		PS_BEACON(0x42);
	}
	// ============================================================ E: down projection
	PS_REFILL_D(l + 1, 0);
	{
		PsRun run;
		if (hasE) {
			run = ps_prepare(pw, (l << 4) | 5, &s_u[3], tmem, &bar_E, par);
			ps_act_quant(pw, (l << 4) | 5, llb + a.ll_act + size_t(s_c.splitE) * a.E.nq * 4, a.E.nq, &s_u[3], bred, &s_xscale);
		}
		if (tid == PS_THREADS - 32 && l + 1 == L) {
			// last layer: the up/gate region is idle until the lm_head, whose ring starts there. Its first stages
			// are requested now, so that they land under the down projection and the final norm.
#pragma unroll 1
			for (int sg = 0; sg < lm_pre; sg++)
				ps_issue(R_D + size_t(sg) * a.lm_stage_bytes, a.lm_tiled + (size_t(cta) * a.lm_nchunk + sg) * a.lm_stage_bytes, uint32_t(a.lm_stage_bytes),
				         &bar_lm[sg], pol, &s_abort);
		}
		PS_STAMP();
		PS_GT(8);
		PS_BEACON(0x51);
		if (hasE) {
			PS_STAMP();
			pm = ps_unit(pw, (l << 4) | 5, run, bar_m, pm, &s_xscale, cta != a.fault_cta ? llb + s_u[3].dst : nullptr, a.lut, lut_s, keep);
			PS_STAMP();
		} else {
			if (tid == 0) ps_st(llb + a.ll_pres + s_c.presE, 0.0f);
			PS_STAMP();
			PS_STAMP();
		}
		PS_STAMP();
		PS_GT(9);
		PS_BEACON(0x52);
	}
	return pm;
}

template <bool DBG>
__global__ void __launch_bounds__(PS_THREADS, 1) decode_persist_kernel(const __grid_constant__ PsArgs a) {
	uint8_t *smem = reinterpret_cast<uint8_t *>((uintptr_t(ps_dyn) + 127) & ~uintptr_t(127));  // the host adds 128 bytes of slack
#pragma unroll 1
	for (int i = threadIdx.x; i < int(sizeof(PsArgs) / 4); i += PS_THREADS) memcpy(reinterpret_cast<char *>(&s_args) + 4 * i, reinterpret_cast<const char *>(&a) + 4 * i, 4);
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int cta = blockIdx.x, G = gridDim.x;
	const int D = a.D, L = a.L;

	if (tid == 0) {
		ps_mbar_init(&bar_A, 1);
		ps_mbar_init(&bar_C, 1);
		ps_mbar_init(&bar_D, 1);
		ps_mbar_init(&bar_E, 1);
#pragma unroll 1
		for (int i = 0; i < 8; i++) {
			ps_mbar_init(&bar_lm[i], 1);
			ps_mbar_init(&emp_lm[i], 1);
		}
#pragma unroll 1
		for (int i = 0; i < PS_TILES; i++) ps_mbar_init(&bar_m[i], 1);
#pragma unroll 1
		for (int i = 0; i < 2; i++) {
			ps_mbar_init(&acc_full[i], 1);
			ps_mbar_init(&acc_free[i], 4);
		}
		s_abort = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == 1) {
		__syncwarp();
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ps_smem(&s_tmem)), "r"(PS_TMEM) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	if (a.lut.size <= PS_LUT)
#pragma unroll 1
		for (int i = tid; i < a.lut.size; i += PS_THREADS) reinterpret_cast<float *>(smem + a.off_lut)[i] = a.lut.table[i];
	{
		// (bytes: an int store to a struct of pointers would be one that the compiler need not see)
#pragma unroll 1
		for (int i = tid; i < L * int(sizeof(PsLayer) / 4); i += PS_THREADS) memcpy(reinterpret_cast<char *>(s_ly) + 4 * i, reinterpret_cast<const char *>(a.layers) + 4 * i, 4);
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const PsW pw{&s_abort, a.err, a.wait_clocks, unsigned(a.poll_ns)};
	uint32_t pm = 0;

	{
		const int uA = cta - a.A.cta0, uC = cta - a.C.cta0, uD = cta - a.Dp.cta0, uE = cta - a.E.cta0;
		const bool hA = uA >= 0 && uA < a.A.units, hC = uC >= 0 && uC < a.C.units, hD = uD >= 0 && uD < a.Dp.units, hE = uE >= 0 && uE < a.E.units;
		if (tid == 0) {
			s_c.tm = *(volatile uint32_t *)&s_tmem;
			s_c.policy_first = ps_evict_first();
			s_c.policy_last = ps_evict_last();
			s_c.splitC = hC ? uC / a.C.ntiles : 0;
			s_c.splitE = hE ? uE / a.E.ntiles : 0;
			s_c.presE = uE < 0 ? cta : cta - a.E.units;  // index of this CTA's presence word (if !hasE)
			// the unit this CTA fetches for a phase of layer l (one lane issues the copy)
			s_c.srcA = a.tiled + a.tl_A + size_t(hA ? uA : 0) * a.A.bytes;
			s_c.srcC = a.tiled + a.tl_C + size_t(hC ? uC : 0) * a.C.bytes;
			s_c.srcD = a.tiled + a.tl_D + size_t(hD ? uD : 0) * a.Dp.bytes;
			s_c.srcE = a.tiled + a.tl_E + size_t(hE ? uE : 0) * a.E.bytes;
			s_c.has = (hA ? 1 : 0) | (hC ? 2 : 0) | (hD ? 4 : 0) | (hE ? 8 : 0);
		}
		if (lane == 0) {
			ps_fill_unit(a.A, &s_u[0], warp, smem_s, a.off_A, a.ll_qkv + (hA ? uA % a.A.ntiles : 0) * a.A.ncol);
			ps_fill_unit(a.C, &s_u[1], warp, smem_s, a.off_C, a.ll_op + (hC ? (uC / a.C.ntiles) * D + (uC % a.C.ntiles) * a.C.ncol : 0));
			ps_fill_unit(a.Dp, &s_u[2], warp, smem_s, a.off_D, a.ll_act + (hD ? uD : 0) * a.Dp.ncol);
			ps_fill_unit(a.E, &s_u[3], warp, smem_s, a.off_E, a.ll_dn + (hE ? (uE / a.E.ntiles) * D + (uE % a.E.ntiles) * a.E.ncol : 0));
			ps_fill_unit(a.lm, &s_u[4], warp, smem_s, a.off_D, 0);
		}
		__syncthreads();
	}
	if (tid == 0) {
		if (hasA) ps_issue(R_A, s_c.srcA, a.A.bytes, &bar_A, pol, &s_abort);
		if (hasC) ps_issue(R_C, s_c.srcC, a.C.bytes, &bar_C, pol, &s_abort);
		if (hasD) ps_issue(R_D, s_c.srcD, a.Dp.bytes, &bar_D, pol, &s_abort);
		if (hasE) ps_issue(R_E, s_c.srcE, a.E.bytes, &bar_E, pol, &s_abort);
	}

	if (tid == 0) s_t = PsLive{0, 0, 0, 0, 0, __ldcg(a.tok), __ldcg(a.next_pos)};
	__syncthreads();
	if (tid == 0) s_dbg_n = 0;
	// ring stages of the lm_head that fit the up/gate region and belong to this CTA's first tile (chunks 0 .. lm_pre - 1)
	int lc = 0;  // layers so far
#pragma unroll 1
	for (int step = 0; step < a.n_steps; step++) {
		const bool more = (step + 1 < a.n_steps);
		const bool dbg_on = DBG && (a.dbg != nullptr) && cta == a.dbg_cta && tid == 0 && !more;
		PS_STAMP();
		// ---------------------------------------------------------------- embedding
		int tok = s_t.tok;
		const int pos = s_t.pos;
		if (a.force_ids) tok = __ldg(a.force_ids + step);
		if (tok < 0 || tok >= a.V) {
			if (tid == 0 && cta == 0) atomicExch(a.err, 1);
			tok = 0;
		}
		// Cache chunks per head of this token's attention: the multiple of 3 with the least 3 * steps + a third of the chunks. A warp holds two
		// rows from before the poll for q|k|v, so a chunk takes a dependent step for every 24 rows; the merge in phase C requests four chunks per
		// group of threads at once (12 a round trip with the 1B plan's three groups, 24 with the 270m plan's six), but every further chunk's CTA
		// also publishes a row, so more chunks than rows ask for cost time: with 24 cached rows 3 chunks take 434 us a token and 24 take 459 (1B; 270m 267 and
		// 273), with 210 12 take 441 and 24 455 (290 and 293). Behind 400 rows the price of a merge in the rule is too high: 24 chunks take 453 us
		// where its 12 take 457 at 400 rows, 455 / 460 at 520 and 470 / 476 at 4096 positions (270m 277 / 281, 282 / 288, 301 / 307).
		if (warp == 0) {
			const bool loc = lane < 16;
			const int n = min(3 * ((lane & 15) + 1), a.nch_max), v = loc ? min(pos + 1, a.slots_local) : min(pos + 1, a.slots_global);
			const int steps = ((v + n - 1) / n + 2 * PS_NW - 1) / (2 * PS_NW);
			const unsigned key = unsigned(3 * steps + (n + 2) / 3) << 8 | unsigned(n);
			const unsigned kl = __reduce_min_sync(0xffffffffu, loc ? key : ~0u), kg = __reduce_min_sync(0xffffffffu, loc ? ~0u : key);
			if ((lane & 15) == 0) {  // position bookkeeping (KVCache, reference decode.hpp:45-70)
				const int given = loc ? a.nch_local : a.nch_global, nch = given ? given : int((loc ? kl : kg) & 255u);
				const int p = loc ? pos : min(pos, a.slots_global - 1);
				if (!loc && pos >= a.slots_global && cta == 0) atomicExch(a.err, 2);
				s_at[loc] = PsSpan{p, loc ? (p - __ldcg(a.ring_base)) % a.slots_local : p, v, nch, (v + nch - 1) / nch};
			}
		}
#pragma unroll 1
		for (int d = tid; d < D; d += PS_THREADS) h[d] = a.wte_s[d] * (a.sqrtD * float(a.wte[size_t(tok) * D + d]));
		__syncthreads();

#pragma unroll 1
		for (int l = 0; l < L; l++, lc++) pm = ps_layer<DBG>(l, lc, more, pm);

		// ================================================================ lm_head
		// (its ring lies over the now idle up/gate and down regions)
		{
			float *const lllast = a.ll + size_t((lc + 2) % 3) * a.ll_stride;
			ps_final_norm(pw, (L << 4) | 6, D, h, &s_u[4], &s_xscale, lllast + a.ll_dn, a.E.nsplit, lllast + a.ll_pres, G - a.E.units,
			           s_ly[L - 1].mlp_post, a.final_norm, keep, cta == 0 ? a.xnorm_out : nullptr);
		}
		PS_STAMP();
		PS_BEACON(0x61);
		const PsLmOut lo = ps_lm_head(a, pw, R_D, smem_s, s_xscale, tmem, bar_lm, emp_lm, acc_full, acc_free, s_t.plm, s_t.pemp, s_t.acc_n, pol, keep, lm_pre);
		__syncthreads();
		if (tid == 0) {
			s_t.acc_n += (a.lm_ntiles - cta + G - 1) / G;
			s_t.plm = lo.plm;
			s_t.pemp = lo.pemp;
		}

		// ================================================================ sampler
		PS_STAMP();
		PS_BEACON(0x70);
		const PsSampOut so = ps_sampler(a, pw, lo.best, lo.best_i, s_t.epoch, s_t.n_logged, wm, s_cdf, s_f, s_i, bred, reinterpret_cast<float *>(R_D));
		PS_STAMP();
		PS_BEACON(0x7F);
		if (tid == 0) {
			s_t.epoch = so.epoch;
			if (a.sampler != 0) s_t.n_logged++;
			s_t.tok = so.tok;
			s_t.pos++;
			if (cta == 0) *a.next_pos = s_t.pos;
		}
		// the ring is idle again: fetch the next token's layer-0 up/gate and down units
		if (tid == 0 && more) {
			if (hasD) ps_issue(R_D, s_c.srcD, a.Dp.bytes, &bar_D, pol, &s_abort);
			if (hasE) ps_issue(R_E, s_c.srcE, a.E.bytes, &bar_E, pol, &s_abort);
		}
		if (__syncthreads_or(*(volatile int *)&s_abort)) break;  // the whole CTA leaves together
	}
	if (*(volatile int *)&s_abort) {
		// gave up: let the bulk copies still in flight land in this CTA's shared memory before it returns
		const long long t0 = clock64();
		while (clock64() - t0 < 400000) {
		}
		__syncthreads();
	}
	tc_fence_before();
	__syncthreads();
	if (warp == 1) {
		__syncwarp();
		tc_fence_after();
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(PS_TMEM) : "memory");
	}
	if (cta == 0 && tid == 0 && a.log_count) *a.log_count = s_t.n_logged;
	// Leave the hand-off arena as the next launch expects it: copy 0 empty (copies 1 and 2 are wiped during
	// its layers 0 and 1, like every copy a layer before its use). Every CTA is past the last token's grid
	// barriers, which all CTAs reach only after their last read of the arena.
	if (!*(volatile int *)&s_abort) {
		float4 *c0 = reinterpret_cast<float4 *>(a.ll);
		const int n4 = a.ll_stride / 4, per = (n4 + G - 1) / G;
		const float e = __uint_as_float(PS_EMPTY);
#pragma unroll 1
		for (int i = cta * per + tid; i < min(n4, (cta + 1) * per); i += PS_THREADS) __stcg(c0 + i, make_float4(e, e, e, e));
	}
}
#undef h
#undef att
#undef smem_s
#undef lut_s
#undef tmem
#undef pol
#undef keep
#undef R_A
#undef R_C
#undef R_D
#undef R_E
#undef PS_REFILL_D
#undef PS_REFILL_E
#undef hasA
#undef hasC
#undef hasD
#undef hasE
#undef lm_pre

}  // namespace tg
