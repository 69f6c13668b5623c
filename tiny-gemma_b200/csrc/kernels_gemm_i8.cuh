// GEMM with int8 weights on the integer tensor cores (tcgen05 kind::i8 + TMEM):
//   C[m, n] = scale[n] * sum_k A[m,k] * W[k,n],  A fp32, W int8 [K,N] row-major
// (gemm::qgemmnn, reference linalg.hpp:210-308, which runs a full-K fp32 FMA chain per output).
//
// Arithmetic: a row of A is written as x = 2^(e-30) * (d3 * 2^24 + d2 * 2^16 + d1 * 2^8 + d0), one exponent e per
// row (2^e > the row's largest |x|), four signed 8-bit digits. An element within a factor 2^7 of the row's largest
// keeps all 24 bits of its fp32 mantissa; below that the representation is still exact to 2^-31 of the largest (the operators
// recompute rows for which that is not enough, see i8_wide). The
// weights go to the tensor cores as they lie in memory, the digit products are summed EXACTLY in int32 (at most
// 6912 * 128 * 128 < 2^31), and only the epilogue rounds: it joins the four sums in fp32. Against three bf16 terms with fp32 accumulation
// (6 bytes per activation, weights converted on the SM, truncating adds): 4 products at twice the bf16 rate instead of
// 3, no conversion of W, and no accumulation error that grows with K, so K is never split for accuracy.
//
// Operand roles are swapped: the MMA's M dimension (128 TMEM lanes) runs over columns of W, its N dimension over
// (token, digit). So the token count pads to 8, not to 128, one MMA of N = 256 covers all four digits of 64 tokens
// against one fetched W tile, and in the epilogue the 32 lanes of a warp hold 32 consecutive columns of one token: a
// store instruction writes 128 contiguous bytes straight from registers.
//
// Operand layouts:
//   W       box of 128 columns x 128 rows by TMA with the 128-byte swizzle = MN-major operand, 8 k-rows per 1 KiB atom
//   digits  [K / 64][groups of 8 tokens][4 digits][8 tokens][64 k] bytes, 64-byte swizzle (K-major operand, 512 B per
//           (group, digit)): a CTA's tokens of one K-block are contiguous, one bulk copy each
// Accumulator column of (group g, digit d, token r): 32 g + 8 d + r.
//
// The kernel is persistent, one CTA per SM walking tiles of 128 columns x up to 64 tokens, with two accumulators of 256
// TMEM columns: the epilogue of a tile (8 warps) and the loads of the next one run under MMAs. One tile per CTA spent
// more time outside its K loop than in it (K = 1152: ~10K of 20K clk: start ~1.5K, first operands ~2.5K, epilogue ~4K).
// A completed mbarrier test costs ~180 clk on this part, so a stage is large: 128 k, 48 KB, 512 clk of MMAs.
// The MMA-issuing and the copying warp run converged: all lanes walk the loop and wait, one elected lane issues, and a
// wait that runs out changes no control flow (it only stops waiting from then on). The operands of these instructions live
// in uniform registers; in a single-lane branch with a conditional exit they are moved there by a loop around every
// instruction. Measured per MMA: 40 clk to issue, 21 for its share of a completed barrier test, against ~260 in a
// lane-0 branch with a break — which made a stage take 580-760 clk instead of 512.
// Two CTAs of a cluster can share a tile of 256 columns (cta_group::2): each holds its own columns and half of the
// digits, which halves the digits' L2 traffic.
//
// All waits are bounded; a wait that runs out sets *err and the CTA drains and frees its TMEM before returning.
#pragma once
#include <cuda.h>

#include <type_traits>

#include "gemm_i8_tiles.h"  // plan, tile walk
#include "kernels_tc.cuh"   // tcgen05 / bulk-copy helpers
#include "tg_common.cuh"

namespace tg {

constexpr int I8_THREADS = 320;                // producer, MMA issuer, 8 epilogue warps
// CG CTAs work on a tile of CG * 128 columns: each holds its own 128 columns of W and 1 / CG of the digits. A stage of the ring holds the digits of SLOT token
// groups. With the few tokens of a decode step four stages that 64 tokens would fit left 64 KB of weights in flight per SM, too few for HBM's rate times its
// latency: three rows of 640 x 262144 35.8 us, with eight small stages 31.4 (1152 rows: 58.6 and 52.9; ncu, single CTAs in both). As constants, or each MMA takes longer to issue (a ring whose
// numbers follow the launch: 77 x 1152 x 6912 18.3 -> 18.8 us). 220 KB in place of 192 leave no room for a CTA of the next launch: a prompt of 61 tokens 1196 -> 1248 us.
constexpr int I8_FEW = 2;                // groups of a tile that takes the small stages
constexpr int I8_ROOM = 192 * 1024, I8_SMEM = I8_ROOM + 1024;
template <int CG, int SLOT> struct I8Shape {
	static constexpr int X_KB = SLOT * I8_GROUP_BYTES / CG;  // digits of one K-block in a CTA
	static constexpr int STAGE = I8_W_BYTES + (I8_SK / I8_BK) * X_KB;
	static constexpr int NST = I8_ROOM / STAGE;
};

// ------------------------------------------------------------------ digits
// exponent of a row from the bits of its largest |x| (NaN and infinity compare above every finite value)
__device__ __forceinline__ int i8_row_exp(uint32_t maxbits) { return max(int(maxbits >> 23) - 126, -96); }
__device__ __forceinline__ float i8_pow2(int e) { return __uint_as_float(uint32_t(e + 127) << 23); }  // -126 <= e <= 127
// what a digit sum is multiplied with: 2^(e - 30), or NaN for a row that holds a NaN or an infinity
__device__ __forceinline__ float i8_row_scale(uint32_t maxbits) {
	return maxbits >= 0x7F800000u ? __uint_as_float(0x7FC00000u) : i8_pow2(i8_row_exp(maxbits) - 30);
}
__device__ __forceinline__ float i8_row_mul(uint32_t maxbits) { return i8_pow2(30 - i8_row_exp(maxbits)); }
__device__ __forceinline__ uint32_t i8_abs_bits(float x) { return __float_as_uint(x) & 0x7FFFFFFFu; }

// byte i of the result = digit i: q = sum d_i 256^i with d_i in [-128, 127] <=> q + 0x80808080 has bytes d_i + 128
__device__ __forceinline__ uint32_t i8_digits(float x, float mul) {
	return (uint32_t(__float2int_rn(x * mul)) + 0x80808080u) ^ 0x80808080u;
}
// byte offset of (row, 4 consecutive k starting at k4 * 4, digit 0) in the packed operand; digits are 512 B apart
__device__ __forceinline__ size_t i8_offset(int row, int k4, int groups) {
	const int kb = k4 >> 4, chunk = (k4 >> 2) & 3, r = row & 7;
	return (size_t(kb) * groups + (row >> 3)) * I8_GROUP_BYTES + r * 64 + ((chunk ^ (r >> 1)) << 4) + ((k4 & 3) << 2);
}
// the digits of four values -> four words of one digit each
__device__ __forceinline__ void i8_transpose4(const uint32_t (&q)[4], uint32_t &d0, uint32_t &d1, uint32_t &d2, uint32_t &d3) {
	const uint32_t ab01 = __byte_perm(q[0], q[1], 0x5140), ab23 = __byte_perm(q[0], q[1], 0x7362);
	const uint32_t cd01 = __byte_perm(q[2], q[3], 0x5140), cd23 = __byte_perm(q[2], q[3], 0x7362);
	d0 = __byte_perm(ab01, cd01, 0x5410);
	d1 = __byte_perm(ab01, cd01, 0x7632);
	d2 = __byte_perm(ab23, cd23, 0x5410);
	d3 = __byte_perm(ab23, cd23, 0x7632);
}
// four consecutive values of a row -> one 4-byte store per digit
__device__ __forceinline__ void i8_pack4(uint8_t *out, int groups, int row, int k4, const float4 &v, float mul) {
	const uint32_t q[4] = {i8_digits(v.x, mul), i8_digits(v.y, mul), i8_digits(v.z, mul), i8_digits(v.w, mul)};
	uint32_t d[4];
	i8_transpose4(q, d[0], d[1], d[2], d[3]);
	uint8_t *p = out + i8_offset(row, k4, groups);
#pragma unroll
	for (int i = 0; i < 4; i++) *reinterpret_cast<uint32_t *>(p + 512 * i) = d[i];
}
__device__ __forceinline__ uint32_t warp_umax(uint32_t v) { return __reduce_max_sync(0xffffffffu, v); }
template <int NW> __device__ __forceinline__ uint32_t block_umax(uint32_t v, uint32_t *red) {
	v = warp_umax(v);
	__syncthreads();
	if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
	__syncthreads();
	uint32_t t = 0;
#pragma unroll
	for (int w = 0; w < NW; w++) t = max(t, red[w]);
	return t;
}

// (The rows that pad M to whole groups of 8 are never written: a token's sums involve no other token, and the sums of
// rows >= M are not stored.)

// Rows that the digits do not hold well enough. An element below 2^-7 of its row's largest loses mantissa bits, and a column
// whose weights on the large elements are zero sees that loss undiluted. Rows in which more than an eighth of the nonzero elements
// (of some warp's part of the row) lie below 2^-12 of the largest (such an element is kept to 2^-19 of itself), and rows below 2^-96
// altogether, are marked by the operators' packing and recomputed by qgemm_wide_rows_kernel. A normal row with one element of s
// sigmas is marked from s = 512 on, from 256 on now and then; below, a column that does not see that element is off by 1.4e-7 at
// most. (A model's own passes mark nothing: their rows come out of a norm or a GeGLU, and its decode steps hold them to 2^-31 of the
// largest in any case.) Called by whole warps; the zeros are told apart only where many elements are small.
template <int PER> __device__ __forceinline__ bool i8_wide(const float4 (&v)[PER], uint32_t maxbits) {
	const float below = __uint_as_float(uint32_t(max(int(maxbits >> 23) - 11, 0)) << 23);
	int small = 0, zero = 0;
#pragma unroll
	for (int j = 0; j < PER; j++) small += (fabsf(v[j].x) < below) + (fabsf(v[j].y) < below) + (fabsf(v[j].z) < below) + (fabsf(v[j].w) < below);
	small = __reduce_add_sync(0xffffffffu, small);
	if (8 * small > 128 * PER) {
#pragma unroll
		for (int j = 0; j < PER; j++) zero += (v[j].x == 0.0f) + (v[j].y == 0.0f) + (v[j].z == 0.0f) + (v[j].w == 0.0f);
		zero = __reduce_add_sync(0xffffffffu, zero);
	}
	const bool tiny = maxbits != 0u && int(maxbits >> 23) - 126 < -96;
	return maxbits < 0x7F800000u && (tiny || 8 * (small - zero) > 128 * PER - zero);
}

// fp32 rows -> digits. One CTA of NT threads per row, the row in registers: K <= NT * 4 * PER.
// WIDE: wide[row] = 1 for a row that the digits do not hold, and *any (host memory) is set.
template <int NT, int PER, bool WIDE>
__global__ void __launch_bounds__(NT) i8_pack_kernel(const float *A, uint8_t *out, float *rowscale, int K, int groups, int *wide, int *any) {
	pdl_trigger();
	pdl_wait();
	__shared__ uint32_t red[NT / 32];
	const int row = blockIdx.x, tid = threadIdx.x;
	float4 v[PER];
	uint32_t mx = 0;
#pragma unroll
	for (int j = 0; j < PER; j++) {
		const int k4 = tid + NT * j;
		v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
		if (4 * k4 < K) v[j] = *reinterpret_cast<const float4 *>(A + size_t(row) * K + 4 * k4);
		mx = max(max(max(mx, i8_abs_bits(v[j].x)), max(i8_abs_bits(v[j].y), i8_abs_bits(v[j].z))), i8_abs_bits(v[j].w));
	}
	mx = block_umax<NT / 32>(mx, red);
	const float mul = i8_row_mul(mx);
	if (tid == 0) rowscale[row] = i8_row_scale(mx);
#pragma unroll
	for (int j = 0; j < PER; j++)
		if (4 * (tid + NT * j) < K) i8_pack4(out, groups, row, tid + NT * j, v[j], mul);
	if (WIDE) {
		const int w = __syncthreads_or(i8_wide(v, mx));
		if (tid == 0) {
			wide[row] = w;
			if (w) *static_cast<volatile int *>(any) = 1;
		}
	}
}

// The marked rows of C = A . W * scales, from the fp32 rows, with products and sums in fp64 (both exact or as good as that):
// 128 columns per CTA, eight warps with every eighth group of four k each (a warp reads 128 contiguous bytes of W per k), eight
// rows at a time, the warps' sums added in order. An ordinary call never launches it (the marking itself: 142.9 -> 144.3 us for
// 4001 rows of 6912 x 1152). Up to eight marked rows add 0.17 ms there, one CTA's chain of loads; 4001 marked rows 5.9 ms, bound by
// the fp64 pipe and the conversions (one k-group of loads in flight: 12.8 ms; four rows at a time: 14.4).
__device__ __forceinline__ double i8_to_double(uint32_t word, int byte) {  // exact: 2^52 + (b + 128) in the mantissa
	return __hiloint2double(0x43300000, int(__byte_perm(word ^ 0x80808080u, 0u, 0x4440u + byte))) - 4503599627370624.0;
}
__global__ void __launch_bounds__(256) qgemm_wide_rows_kernel(float *C, const float *A, const int8_t *W, const float *scales, const int *wide, int M, int K, int N) {
	pdl_trigger();
	pdl_wait();
	constexpr int R = 8, H = 4;  // rows at a time, rows whose sums meet at a time
	__shared__ int list[256], count[8];
	__shared__ double part[8][H][128];
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n0 = blockIdx.x * 128;
	const int chunk = (M + gridDim.y - 1) / gridDim.y, r0 = blockIdx.y * chunk, r1 = min(M, r0 + chunk);
	for (int base = r0; base < r1; base += 256) {
		__syncthreads();
		const bool mine = base + tid < r1 && wide[base + tid] != 0;
		const unsigned m = __ballot_sync(0xffffffffu, mine);
		if (lane == 0) count[warp] = __popc(m);
		__syncthreads();
		int n = 0, at = __popc(m & ((1u << lane) - 1u));
		for (int w = 0; w < 8; w++) {
			if (w < warp) at += count[w];
			n += count[w];
		}
		if (mine) list[at] = base + tid;
		__syncthreads();
		for (int first = 0; first < n; first += R) {
			const float *row[R];
#pragma unroll
			for (int i = 0; i < R; i++) row[i] = A + size_t(list[min(first + i, n - 1)]) * K;
			double acc[R][4] = {};
#pragma unroll 2
			for (int k = 4 * warp; k < K; k += 32) {
				uint32_t w[4];
#pragma unroll
				for (int q = 0; q < 4; q++) w[q] = *reinterpret_cast<const uint32_t *>(W + size_t(k + q) * N + n0 + 4 * lane);
				float4 x[R];
#pragma unroll
				for (int i = 0; i < R; i++) x[i] = *reinterpret_cast<const float4 *>(row[i] + k);
#pragma unroll
				for (int q = 0; q < 4; q++) {
					const double w0 = i8_to_double(w[q], 0), w1 = i8_to_double(w[q], 1), w2 = i8_to_double(w[q], 2), w3 = i8_to_double(w[q], 3);
#pragma unroll
					for (int i = 0; i < R; i++) {
						const double xi = q == 0 ? x[i].x : (q == 1 ? x[i].y : (q == 2 ? x[i].z : x[i].w));
						acc[i][0] = fma(xi, w0, acc[i][0]);
						acc[i][1] = fma(xi, w1, acc[i][1]);
						acc[i][2] = fma(xi, w2, acc[i][2]);
						acc[i][3] = fma(xi, w3, acc[i][3]);
					}
				}
			}
#pragma unroll
			for (int h = 0; h < R; h += H) {
				__syncthreads();  // (the sums before have been read)
#pragma unroll
				for (int i = 0; i < H; i++)
#pragma unroll
					for (int c = 0; c < 4; c++) part[warp][i][4 * lane + c] = acc[h + i][c];
				__syncthreads();
				for (int q = tid; q < min(H, n - first - h) * 128; q += 256) {
					const int i = q >> 7, c = q & 127;
					double s = 0.0;
#pragma unroll
					for (int w = 0; w < 8; w++) s += part[w][i][c];
					C[size_t(list[first + h + i]) * N + n0 + c] = float(s * double(scales[n0 + c]));
				}
			}
		}
	}
}

// Residual + sandwich norms of one row, fused with the operand packing of the next GEMM:
//   if t:     h += rmsnorm(t; w_post)        (reference modules.hpp: post-norm, then the residual add)
//   if w_pre: pack( rmsnorm(h; w_pre) )      (the pre-norm of the following matmuls)
// t is the partial sums of the GEMM before: t[d] = tscale[d] * sum_sp t[(sp * M + row) * dim + d], added in split order.
// A row belongs to NT threads, its values stay in their registers (dim <= 4 * NT * PER). A row is a chain of dependent
// round trips (loads, two reductions), so everything that does not depend on the partial sums is requested before them.
//   NT = 160, 288 (one CTA per row, a quad of values per thread): a few hundred rows, all resident at once, the chain's length
//   counts, and with it the instructions: rows of 1152 took 3.1 us with two quads per thread, half of them idle, and the column scales requested late
//   NT = 32  (one warp per row, 8 rows per CTA): thousands of rows; no barriers, shuffles only, more rows in flight
template <int NT, int PER>
__global__ void __launch_bounds__(NT == 32 ? 256 : NT) resnorm_i8_kernel(float *h, const float *t, const float *w_post, const float *w_pre, uint8_t *out,
                                                                         float *rowscale, int M, int dim, int groups, int nsplit,
                                                                         const float *tscale) {
	constexpr int NW = NT / 32;
	__shared__ float2 red[2][NT == 32 ? 1 : NW];  // (one per reduction: a barrier each)
	const int lt = NT == 32 ? int(threadIdx.x & 31) : int(threadIdx.x);
	const int row = NT == 32 ? int(blockIdx.x * 8 + (threadIdx.x >> 5)) : int(blockIdx.x);
	const int n4 = dim / 4;
	// sum of a, maximum of the bit patterns b over the row's threads; i: the first or the second reduction
	auto reduce = [&](float a, uint32_t b, int i) -> float2 {
		a = warp_sum(a);
		b = warp_umax(b);
		if (NT == 32) return make_float2(a, __uint_as_float(b));
		if ((threadIdx.x & 31) == 0) red[i][threadIdx.x >> 5] = make_float2(a, __uint_as_float(b));
		__syncthreads();
		float s = 0.0f;
		uint32_t m = 0;
#pragma unroll
		for (int w = 0; w < NW; w++) {
			s += red[i][w].x;
			m = max(m, __float_as_uint(red[i][w].y));
		}
		return make_float2(s, __uint_as_float(m));
	};
	const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
	float4 wpost[PER], wpre[PER], scl[PER];  // the weights are nobody's output: requested before the wait for the predecessor
#pragma unroll
	for (int j = 0; j < PER; j++) {
		const int k4 = lt + NT * j;
		wpost[j] = wpre[j] = scl[j] = z4;
		if (NT != 32 && k4 < n4) {
			if (t) wpost[j] = __ldg(reinterpret_cast<const float4 *>(w_post) + k4);
			if (t) scl[j] = __ldg(reinterpret_cast<const float4 *>(tscale) + k4);
			if (w_pre) wpre[j] = __ldg(reinterpret_cast<const float4 *>(w_pre) + k4);
		}
	}
	pdl_trigger();
	pdl_wait();
	if (row >= M) return;  // (whole warps)
	float4 *hrow = reinterpret_cast<float4 *>(h + size_t(row) * dim);
	float4 hv[PER];
#pragma unroll
	for (int j = 0; j < PER; j++) {
		const int k4 = lt + NT * j;
		hv[j] = z4;
		if (k4 < n4) hv[j] = hrow[k4];
	}
	if (t) {
		float4 acc[PER];
#pragma unroll
		for (int j = 0; j < PER; j++) acc[j] = z4;
		const float4 *base = reinterpret_cast<const float4 *>(t + size_t(row) * dim);
		const size_t stride = size_t(M) * n4;
		auto splits = [&](auto qb, int s0) {  // qb splits requested together
			constexpr int QB = decltype(qb)::value;
			float4 q[QB][PER];
#pragma unroll
			for (int i = 0; i < QB; i++)
#pragma unroll
				for (int j = 0; j < PER; j++) {
					const int k4 = lt + NT * j;
					q[i][j] = z4;
					if (k4 < n4 && s0 + i < nsplit) q[i][j] = base[size_t(s0 + i) * stride + k4];
				}
#pragma unroll
			for (int i = 0; i < QB; i++)
#pragma unroll
				for (int j = 0; j < PER; j++) {
					acc[j].x += q[i][j].x; acc[j].y += q[i][j].y; acc[j].z += q[i][j].z; acc[j].w += q[i][j].w;
				}
		};
		if (NT == 32 || PER > 2) {
			for (int s0 = 0; s0 < nsplit; s0++) splits(std::integral_constant<int, 1>(), s0);
		} else if (nsplit <= 4) {
			splits(std::integral_constant<int, 4>(), 0);
		} else if (PER == 1 && nsplit > 8) {
			for (int s0 = 0; s0 < nsplit; s0 += 16) splits(std::integral_constant<int, PER == 1 ? 16 : 8>(), s0);
		} else {
			for (int s0 = 0; s0 < nsplit; s0 += 8) splits(std::integral_constant<int, 8>(), s0);
		}
		float ss = 0.0f;
#pragma unroll
		for (int j = 0; j < PER; j++) {
			const int k4 = lt + NT * j;
			if (k4 < n4) {
				const float4 s4 = NT == 32 ? __ldg(reinterpret_cast<const float4 *>(tscale) + k4) : scl[j];
				acc[j].x *= s4.x; acc[j].y *= s4.y; acc[j].z *= s4.z; acc[j].w *= s4.w;
				ss = fmaf(acc[j].x, acc[j].x, ss);
				ss = fmaf(acc[j].y, acc[j].y, ss);
				ss = fmaf(acc[j].z, acc[j].z, ss);
				ss = fmaf(acc[j].w, acc[j].w, ss);
			}
		}
		const float r = inv_rms(reduce(ss, 0u, 0).x, dim);
#pragma unroll
		for (int j = 0; j < PER; j++) {
			const int k4 = lt + NT * j;
			if (k4 < n4) {
				const float4 w4 = NT == 32 ? __ldg(reinterpret_cast<const float4 *>(w_post) + k4) : wpost[j];
				hv[j].x += (acc[j].x * r) * (w4.x + 1.0f);
				hv[j].y += (acc[j].y * r) * (w4.y + 1.0f);
				hv[j].z += (acc[j].z * r) * (w4.z + 1.0f);
				hv[j].w += (acc[j].w * r) * (w4.w + 1.0f);
				hrow[k4] = hv[j];
			}
		}
	}
	if (!w_pre) return;
	// sum of squares, and the largest |h * (w + 1)|: times the norm factor it bounds the row that is packed
	float ss = 0.0f;
	uint32_t mx = 0;
#pragma unroll
	for (int j = 0; j < PER; j++) {
		const int k4 = lt + NT * j;
		if (NT == 32 && k4 < n4) wpre[j] = __ldg(reinterpret_cast<const float4 *>(w_pre) + k4);
		ss = fmaf(hv[j].x, hv[j].x, ss);
		ss = fmaf(hv[j].y, hv[j].y, ss);
		ss = fmaf(hv[j].z, hv[j].z, ss);
		ss = fmaf(hv[j].w, hv[j].w, ss);
		mx = max(mx, max(max(i8_abs_bits(hv[j].x * (wpre[j].x + 1.0f)), i8_abs_bits(hv[j].y * (wpre[j].y + 1.0f))),
		                 max(i8_abs_bits(hv[j].z * (wpre[j].z + 1.0f)), i8_abs_bits(hv[j].w * (wpre[j].w + 1.0f)))));
	}
	const float2 sm = reduce(ss, mx, 1);
	const float r = inv_rms(sm.x, dim);
	const uint32_t mb = i8_abs_bits(sm.y * r);
	const float mul = i8_row_mul(mb);
	if (lt == 0) rowscale[row] = i8_row_scale(mb);
#pragma unroll
	for (int j = 0; j < PER; j++) {
		const int k4 = lt + NT * j;
		if (k4 < n4)
			i8_pack4(out, groups, row, k4,
			         make_float4((hv[j].x * r) * (wpre[j].x + 1.0f), (hv[j].y * r) * (wpre[j].y + 1.0f), (hv[j].z * r) * (wpre[j].z + 1.0f),
			                     (hv[j].w * r) * (wpre[j].w + 1.0f)),
			         mul);
	}
}

// GeGLU fused with the packing of the down projection's operand: pack( lut(gate) * up ). ug: partial sums of the grouped
// up|gate GEMM (rows of 2I: up columns, then gate columns), su / sg their column scales. One CTA of NT threads per row,
// the row's products in registers (I <= 4 * NT * PER): their largest is needed before the first can be packed. A table of
// up to GE_LUT entries is looked up in shared memory (32 lanes, 32 banks); through the L1 a gather of 32 entries
// touches ~20 of the table's 32 lines, one after the other, which alone took 0.25 ms of 0.58 for 16384 x 6912.
constexpr int GE_LUT = 2048;
// lut(g * gs) * (u * us) of four columns: GeluLut::index, the four look-ups together and selected instead of branched on (int(x) >= 0
// is x > -1; a branch per look-up made 3.6 us of 178 rows of 6912)
__device__ __forceinline__ float4 ge_quad(const GeluLut &lut, const float *values, const float4 &g, const float4 &gs, const float4 &u, const float4 &us) {
	const float v[4] = {g.x * gs.x, g.y * gs.y, g.z * gs.z, g.w * gs.w};
	float x[4], y[4];
	if (lut.inv != 0.0f) {
		const float base = -(lut.mn * lut.inv);
#pragma unroll
		for (int i = 0; i < 4; i++) x[i] = fmaf(v[i], lut.inv, base);
	} else {
#pragma unroll
		for (int i = 0; i < 4; i++) x[i] = (v[i] - lut.mn) / lut.eps;
	}
#pragma unroll
	for (int i = 0; i < 4; i++) y[i] = values[min(max(int(x[i]), 0), lut.size - 1)];
#pragma unroll
	for (int i = 0; i < 4; i++) {
		const float in = int(x[i]) < lut.size ? y[i] : v[i];
		y[i] = x[i] > -1.0f && x[i] < 2147483648.0f ? in : 0.0f;
	}
	return make_float4(y[0] * (u.x * us.x), y[1] * (u.y * us.y), y[2] * (u.z * us.z), y[3] * (u.w * us.w));
}
// CTAS: per SM. With two, 80 bytes of a thread's registers spill (PER = 3). With one, the scales of a thread's columns are requested before the wait for the predecessor (48 rows of 6912, a layer 1.5 us less).
template <int NT, int PER, int CTAS = 2>
__global__ void __launch_bounds__(NT, CTAS) geglu_i8_kernel(const float *ug, uint8_t *out, float *rowscale, int M, int I, int groups, GeluLut lut,
                                                      int nsplit, const float *su, const float *sg) {
	__shared__ uint32_t red[NT / 32];
	__shared__ float table[GE_LUT];
	const int tid = threadIdx.x, n4 = I / 4;
	const bool in_smem = lut.size <= GE_LUT;
	if (in_smem)
		for (int i = tid; i < lut.size; i += NT) table[i] = lut.table[i];
	const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
	float4 fs0 = z4, gs0 = z4;
	if (PER == 1) {  // (nobody's output: requested before the wait; beside a second CTA more of them would not fit the registers)
		fs0 = __ldg(reinterpret_cast<const float4 *>(su) + min(tid, n4 - 1));
		gs0 = __ldg(reinterpret_cast<const float4 *>(sg) + min(tid, n4 - 1));
	}
	float4 fsk[CTAS == 1 ? PER : 1], gsk[CTAS == 1 ? PER : 1];
	if constexpr (CTAS == 1) {
#pragma unroll
		for (int j = 0; j < PER; j++) {
			fsk[j] = __ldg(reinterpret_cast<const float4 *>(su) + min(tid + NT * j, n4 - 1));
			gsk[j] = __ldg(reinterpret_cast<const float4 *>(sg) + min(tid + NT * j, n4 - 1));
		}
	}
	__syncthreads();
	pdl_trigger();
	pdl_wait();
	const float *const values = in_smem ? table : lut.table;
	const size_t stride = size_t(M) * 2 * n4;
	for (int row = blockIdx.x; row < M; row += gridDim.x) {
		const float4 *base = reinterpret_cast<const float4 *>(ug + size_t(row) * 2 * I);
		float4 u[PER], g[PER];
#pragma unroll
		for (int j = 0; j < PER; j++) {
			const int k4 = tid + NT * j;
			u[j] = g[j] = z4;
			if (k4 < n4) {
				u[j] = base[k4];
				g[j] = base[n4 + k4];
			}
		}
		for (int s = 1; s < nsplit; s++) {
			const float4 *bs = base + size_t(s) * stride;
			float4 a[PER], b[PER];
#pragma unroll
			for (int j = 0; j < PER; j++) {
				const int k4 = tid + NT * j;
				a[j] = b[j] = z4;
				if (k4 < n4) {
					a[j] = bs[k4];
					b[j] = bs[n4 + k4];
				}
			}
#pragma unroll
			for (int j = 0; j < PER; j++) {
				u[j].x += a[j].x; u[j].y += a[j].y; u[j].z += a[j].z; u[j].w += a[j].w;
				g[j].x += b[j].x; g[j].y += b[j].y; g[j].z += b[j].z; g[j].w += b[j].w;
			}
		}
		uint32_t mx = 0;
#pragma unroll
		for (int j = 0; j < PER; j++) {
			const int k4 = min(tid + NT * j, n4 - 1);
			float4 fs, gs;
			if constexpr (CTAS == 1) {
				fs = fsk[j];
				gs = gsk[j];
			} else {
				fs = PER == 1 ? fs0 : __ldg(reinterpret_cast<const float4 *>(su) + k4);
				gs = PER == 1 ? gs0 : __ldg(reinterpret_cast<const float4 *>(sg) + k4);
			}
			u[j] = ge_quad(lut, values, g[j], gs, u[j], fs);
			mx = max(mx, max(max(i8_abs_bits(u[j].x), i8_abs_bits(u[j].y)), max(i8_abs_bits(u[j].z), i8_abs_bits(u[j].w))));
		}
		mx = block_umax<NT / 32>(mx, red);
		const float mul = i8_row_mul(mx);
		if (tid == 0) rowscale[row] = i8_row_scale(mx);
#pragma unroll
		for (int j = 0; j < PER; j++)
			if (tid + NT * j < n4) i8_pack4(out, groups, row, tid + NT * j, u[j], mul);
	}
}

// The same for a thousand rows or so of few columns (a 2048-column model's) whose sums are not split, where the GEMM's epilogue does not
// multiply them (launch_gemm_geglu): the rows of a CTA arrive by bulk copies in a ring of STAGES rows, so that loads are in
// flight while a row waits at its barriers and is packed. HBM bounds it.
template <int NT, int PER, int STAGES>
__global__ void __launch_bounds__(NT) geglu_i8_stream_kernel(const float *ug, uint8_t *out, float *rowscale, int M, int I, int groups, GeluLut lut,
                                                             const float *su, const float *sg, int *err) {
	extern __shared__ __align__(128) uint8_t ge_rows[];
	__shared__ uint32_t red[NT / 32];
	__shared__ float table[GE_LUT];
	__shared__ uint64_t full[STAGES];
	const int tid = threadIdx.x, n4 = I / 4;
	const uint32_t row_bytes = uint32_t(I) * 8u;
	const bool in_smem = lut.size <= GE_LUT;
	if (tid == 0) {
		for (int i = 0; i < STAGES; i++) mbar_init(&full[i], 1);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (in_smem)
		for (int i = tid; i < lut.size; i += NT) table[i] = lut.table[i];
	float4 fs[PER], gs[PER];  // (a thread's columns are the same in every row; the L1 beside the ring does not hold the scales)
#pragma unroll
	for (int j = 0; j < PER; j++) {
		const int k4 = min(tid + NT * j, n4 - 1);
		fs[j] = __ldg(reinterpret_cast<const float4 *>(su) + k4);
		gs[j] = __ldg(reinterpret_cast<const float4 *>(sg) + k4);
	}
	__syncthreads();
	pdl_trigger();
	pdl_wait();
	const float *const values = in_smem ? table : lut.table;
	auto issue = [&](int i, int st) {  // the CTA's i-th row; warp 0, converged
		const int row = blockIdx.x + i * gridDim.x;
		if (row < M && tc_elect()) {
			fence_proxy_async();
			mbar_expect_tx(&full[st], row_bytes);
			bulk_load(ge_rows + size_t(st) * row_bytes, ug + size_t(row) * 2 * I, row_bytes, &full[st]);
		}
	};
	if (tid < 32)
		for (int i = 0; i < STAGES; i++) issue(i, i);
	int st = 0;
	uint32_t ph = 0;
	for (int row = blockIdx.x, i = 0; row < M; row += gridDim.x, i++) {
		tc_wait(&full[st], ph, err);
		const float4 *u4 = reinterpret_cast<const float4 *>(ge_rows + size_t(st) * row_bytes), *g4 = u4 + n4;
		float4 v[PER];
		uint32_t mx = 0;
#pragma unroll
		for (int j = 0; j < PER; j++) {
			const int k4 = min(tid + NT * j, n4 - 1);
			const float4 u = u4[k4], g = g4[k4];
			v[j] = ge_quad(lut, values, g, gs[j], u, fs[j]);
			mx = max(mx, max(max(i8_abs_bits(v[j].x), i8_abs_bits(v[j].y)), max(i8_abs_bits(v[j].z), i8_abs_bits(v[j].w))));
		}
		mx = block_umax<NT / 32>(mx, red);  // (its barriers: every thread has read the row)
		if (tid < 32) issue(i + STAGES, st);
		if (++st == STAGES) {
			st = 0;
			ph ^= 1;
		}
		const float mul = i8_row_mul(mx);
		if (tid == 0) rowscale[row] = i8_row_scale(mx);
#pragma unroll
		for (int j = 0; j < PER; j++)
			if (tid + NT * j < n4) i8_pack4(out, groups, row, tid + NT * j, v[j], mul);
	}
}

// ------------------------------------------------------------------ GEMM
struct GemmI8Args : I8Walk {
	const uint8_t *x;       // packed digits
	const float *rowscale;  // [8 * groups]
	// matrix g of the walk has the columns col0[g].. of a partial-sum row (N = all columns)
	int col0[3];
	int ncols[3];            // N_g (a multiple of 128: the last tile of a pair may have only its first half)
	const float *scales[3];  // [N_g]
	float *C[3];             // [M] rows of ldc[g] floats (finished result)
	int ldc[3];
	float *partial;          // [nsplit][M][N] sums without the column scales (raw, or nsplit > 1)
	int M, N;
	int raw;                 // 1: partial sums even unsplit; the consumer adds the splits and applies the column scales
	int w_stream;            // 1: W is read by few CTAs: L2 evict-first
	unsigned long long *top1;  // non-null (nsplit == 1): no C; per token the largest scaled value and its column, as a key
	int top1_col0;
	int *err;
};
// The table's 24 bytes are arguments of the kernel alone that looks up: with 760 bytes of arguments (four tensor maps in front) instead of
// 736 a launch outside a graph took 0.5 to 0.9 us longer (as a call, 77 x 1152 x 6912 19.9 us instead of 19.0, 1500 x 1152 x 1024 23.4
// instead of 22.7; with 888 bytes as with 760).
struct GemmI8GluArgs : GemmI8Args {
	GeluLut lut;
};
enum I8Epilogue { I8_SUMS, I8_GLU, I8_TOP1 };  // finished values or raw sums; the product of up and gate; a key per token
template <I8Epilogue EPI> using I8KernelArgs = std::conditional_t<EPI == I8_GLU, GemmI8GluArgs, GemmI8Args>;
static_assert(4 * sizeof(CUtensorMap) + sizeof(GemmI8Args) <= 736, "see GemmI8GluArgs");

// W tile [128 k][128 n], 128-byte swizzle: MN-major operand; 1 KiB from one group of 8 k-rows to the next
__device__ __forceinline__ uint64_t i8_desc_w(uint32_t addr) {
	return uint64_t((addr & 0x3FFFF) >> 4) | (uint64_t(1) << 16) | (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61);
}
// digits, 64-byte swizzle: K-major operand; 512 B from one group of 8 rows (group, digit) to the next
__device__ __forceinline__ uint64_t i8_desc_x(uint32_t addr) {
	return uint64_t((addr & 0x3FFFF) >> 4) | (uint64_t(1) << 16) | (uint64_t(512 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(4) << 61);
}
// D int32, A and B signed 8 bit, A MN-major (bit 15), B K-major, M = 128 * CG, N = n
template <int CG> __device__ __forceinline__ uint32_t i8_idesc(int n) {
	return (2u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (uint32_t(n >> 3) << 17) | (uint32_t(8 * CG) << 24);
}
template <int CG> __device__ __forceinline__ void i8_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
	if constexpr (CG == 1)
		asm volatile(
		    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
		    "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
		    "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
		    : "memory");
	else
		asm volatile(
		    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
		    "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
		    "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
		    : "memory");
}
// arrives (in both CTAs of a pair) when the MMAs issued so far have completed
template <int CG> __device__ __forceinline__ void i8_commit(uint64_t *bar) {
	if constexpr (CG == 1)
		tc_commit(bar);
	else
		asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"(uint16_t(3))
		             : "memory");
}
// the same barrier in the pair's first CTA
__device__ __forceinline__ uint32_t i8_leader(const void *p) {
	uint32_t r;
	asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(0));
	return r;
}
// box at (x, y) of a tensor map -> this CTA's shared memory, completing on a barrier of the pair's first CTA
__device__ __forceinline__ void i8_pair_load(void *dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
	asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
	             "l"(map), "r"(x), "r"(y), "r"(bar)
	             : "memory");
}
__device__ __forceinline__ void i8_cluster_sync() {
	asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

// xmap (CG = 2): the digits as rows of 512 bytes (one (group, digit) of a K-block), box of 2 * tg rows
//
// GLU: matrix 0 is up, matrix 1 gate, of the same size; the walk is one matrix's and every tile of it is done twice in a row, up and
// then gate. A thread keeps its 32 up values in registers and leaves lut(gate) * up: one column of products goes through memory instead
// of two of sums, and the launch behind it is a plain packing. 4096 x 1152 x (6912 | 6912): 164 us + 68 for the GeGLU -> 184 + 32. The
// epilogue bounds it: with a branch per look-up it took 215 us, and with the table index in a loop of its own as well (GeluLut::index) 250.
// What the epilogue does is a parameter of the kernel, not of the launch: with the code of the others beside it
// a prompt of 178 tokens took 1.79 ms instead of 1.76 (156 registers instead of 140, and more code to fetch).
template <int CG, I8Epilogue EPI, int SLOT = I8_TG>
__global__ void __launch_bounds__(I8_THREADS, 1) qgemm_i8_kernel(const __grid_constant__ CUtensorMap wmap0,
                                                                 const __grid_constant__ CUtensorMap wmap1,
                                                                 const __grid_constant__ CUtensorMap wmap2,
                                                                 const __grid_constant__ CUtensorMap xmap, I8KernelArgs<EPI> a) {
	using SH = I8Shape<CG, SLOT>;
	constexpr int NST = SH::NST;
	constexpr bool GLU = EPI == I8_GLU, TOP1 = EPI == I8_TOP1;
	GeluLut lut{};
	if constexpr (GLU) lut = a.lut;
	pdl_trigger();
	extern __shared__ uint8_t i8_smem_raw[];
	uint8_t *smem = reinterpret_cast<uint8_t *>((uintptr_t(i8_smem_raw) + 1023) & ~uintptr_t(1023));
	__shared__ uint64_t full_bar[NST];  // W and digits of the stage landed
	__shared__ uint64_t free_bar[NST];  // the MMAs that read the stage have completed
	__shared__ uint64_t acc_full[2];        // the accumulator's MMAs have completed
	__shared__ uint64_t acc_free[2];        // the 8 epilogue warps (of both CTAs) have read the accumulator
	__shared__ uint64_t drain_bar;          // every MMA issued has completed
	__shared__ uint32_t tmem_base_s;
	__shared__ int s_fail, s_issued;
	__shared__ float table[GLU ? GE_LUT : 1];

	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int rank = CG == 1 ? 0 : int(blockIdx.x & 1), first = int(blockIdx.x) / CG, stride = int(gridDim.x) / CG;
	// the n-th tile of this CTA or pair
	auto has_tile = [&](int n) { return first + (GLU ? n >> 1 : n) * stride < a.tiles; };
	auto tile = [&](int n) {
		I8Tile t = i8_tile<CG>(a, first + (GLU ? n >> 1 : n) * stride);
		if (GLU) t.grp = n & 1;
		return t;
	};
	if (GLU && lut.size <= GE_LUT)
		for (int i = tid; i < lut.size; i += I8_THREADS) table[i] = lut.table[i];
	if (tid == 0) {
		for (int s = 0; s < NST; s++) {
			mbar_init(&full_bar[s], 1);
			mbar_init(&free_bar[s], 1);
		}
		for (int b = 0; b < 2; b++) {
			mbar_init(&acc_full[b], 1);
			mbar_init(&acc_free[b], 8 * CG);
		}
		mbar_init(&drain_bar, 1);
		s_fail = 0;
		s_issued = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == 1) {
		if constexpr (CG == 1) {
			asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512)
			             : "memory");
			asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
		} else {
			asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512)
			             : "memory");
			asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
		}
	}
	tc_fence_before();
	__syncthreads();
	if constexpr (CG == 2) i8_cluster_sync();  // the barriers of both CTAs are ready
	tc_fence_after();
	const uint32_t tmem_base = tmem_base_s;

	if (warp == 0) {
		// ------------------------------------------------------------ producer
		const uint64_t pol = l2_evict_first_policy();
		auto load_w = [&](const I8Tile &t, int st, int s) {
			const CUtensorMap *wmap = t.grp == 0 ? &wmap0 : (t.grp == 1 ? &wmap1 : &wmap2);
			uint8_t *dst = smem + size_t(s) * SH::STAGE;
			const int y = (t.s0 + st) * I8_SK;
			if constexpr (CG == 2) {
				// (a pair's box is always a whole tile's: what lies past the last token or column is not used)
				if (rank == 0) mbar_expect_tx(&full_bar[s], 2u * I8_W_BYTES + uint32_t(a.tg) * (I8_SK / I8_BK) * I8_GROUP_BYTES);
				i8_pair_load(dst, wmap, t.n0 + 128 * rank, y, i8_leader(&full_bar[s]));
			} else {
				mbar_expect_tx(&full_bar[s], uint32_t(I8_W_BYTES) + uint32_t(t.ng) * (I8_SK / I8_BK) * I8_GROUP_BYTES);
				if (a.w_stream)
					tma_load_2d(dst, wmap, t.n0, y, &full_bar[s], pol);
				else
					tma_load_2d(dst, wmap, t.n0, y, &full_bar[s]);
			}
		};
		auto load_x = [&](const I8Tile &t, int st, int s) {
			uint8_t *dst = smem + size_t(s) * SH::STAGE + I8_W_BYTES;
			const int kb = (t.s0 + st) * (I8_SK / I8_BK);
#pragma unroll
			for (int q = 0; q < I8_SK / I8_BK; q++) {
				if constexpr (CG == 2)
					i8_pair_load(dst + q * SH::X_KB, &xmap, 0, ((kb + q) * a.groups + t.g0) * 4 + rank * 2 * t.ng, i8_leader(&full_bar[s]));
				else
					bulk_load(dst + q * SH::X_KB, a.x + (size_t(kb + q) * a.groups + t.g0) * I8_GROUP_BYTES, uint32_t(t.ng) * I8_GROUP_BYTES, &full_bar[s]);
			}
		};
		int cap = TC_SPIN_CAP, c = 0, s = 0;  // stages issued so far, next slot
		uint32_t ph = 1;                      // parity whose completion frees the slot (a fresh barrier passes parity 1)
		I8Tile t = tile(0);
		// The weights are nobody's output: the first tiles are requested before the wait for the predecessor.
		const int pre = first < a.tiles ? min(NST, t.ns) : 0;
		for (int st = 0; st < pre; st++)
			if (tc_elect()) load_w(t, st, st);
		pdl_wait();
		for (int it = 0; has_tile(it); it++) {
			t = tile(it);
			for (int st = 0; st < t.ns; st++) {
				tc_wait_cap(&free_bar[s], ph, cap);
				if (tc_elect()) {
					if (c >= pre) load_w(t, st, s);
					load_x(t, st, s);
				}
				c++;
				if (++s == NST) {
					s = 0;
					ph ^= 1;
				}
			}
		}
		if (cap == 0 && lane == 0) {
			*static_cast<volatile int *>(a.err) = 6;
			s_fail = 1;
		}
		if (lane == 0) s_issued = c;
	} else if (warp == 1) {
		// ------------------------------------------------------------ MMA issuer (of a pair: the first CTA's)
		if (rank == 0) {
			int cap = TC_SPIN_CAP, s = 0;
			uint32_t ph = 0;
			for (int it = 0; has_tile(it); it++) {
				const I8Tile t = tile(it);
				const uint32_t d = tmem_base + uint32_t(it & 1) * 256, id = i8_idesc<CG>(32 * t.ng);
				tc_wait_cap(&acc_free[it & 1], ((it >> 1) & 1) ^ 1, cap);  // (the first use of a fresh barrier passes)
				for (int st = 0; st < t.ns; st++) {
					tc_wait_cap(&full_bar[s], ph, cap);
					tc_fence_after();
					const uint32_t w = smem_u32(smem) + uint32_t(s) * SH::STAGE;
					const uint64_t dw = i8_desc_w(w), dx = i8_desc_x(w + I8_W_BYTES);
					if (tc_elect()) {
#pragma unroll
						for (int j = 0; j < I8_SK / 32; j++)
							i8_mma<CG>(d, dw + uint64_t(j * 256), dx + uint64_t(((j >> 1) * SH::X_KB + (j & 1) * 32) >> 4), id, (st > 0 || j > 0) ? 1u : 0u);
						i8_commit<CG>(&free_bar[s]);
						if (st == t.ns - 1) i8_commit<CG>(&acc_full[it & 1]);
					}
					__syncwarp();
					if (++s == NST) {
						s = 0;
						ph ^= 1;
					}
				}
			}
			if (tc_elect()) i8_commit<CG>(&drain_bar);
			if (cap == 0 && lane == 0) {
				*static_cast<volatile int *>(a.err) = 6;
				s_fail = 1;
			}
		}
	} else {
		// ------------------------------------------------------------ epilogue (warps 2..9)
		pdl_wait();  // the row scales are the predecessor's output, and C may be its input
		const int quad = warp & 3, sub = (warp - 2) >> 2;  // TMEM lanes 32 * quad ..; two warps share them
		const bool fin = a.nsplit.d == 1 && !a.raw;
		const float *const lut_values = GLU && lut.size <= GE_LUT ? table : lut.table;
		const float lut_base = -(lut.mn * lut.inv);
		float kept[GLU ? 32 : 1];  // GLU: the up values of the tile before
		for (int it = 0; has_tile(it); it++) {
			const I8Tile t = tile(it);
			const float *const scg = t.grp == 0 ? a.scales[0] : (t.grp == 1 ? a.scales[1] : a.scales[2]);
			float *const Cg = t.grp == 0 ? a.C[0] : (t.grp == 1 ? a.C[1] : a.C[2]);
			const size_t ld = fin ? size_t(t.grp == 0 ? a.ldc[0] : (t.grp == 1 ? a.ldc[1] : a.ldc[2])) : size_t(a.N);
			const int pcol = t.grp == 0 ? a.col0[0] : (t.grp == 1 ? a.col0[1] : a.col0[2]);
			const int nl = t.n0 + 128 * rank + quad * 32 + lane;  // this lane's column
			const int ncg = t.grp == 0 ? a.ncols[0] : (t.grp == 1 ? a.ncols[1] : a.ncols[2]);
			const bool live = CG == 1 || t.n0 + 128 * rank < ncg;  // (a pair's last tile may have only its first half)
			float *dst = fin ? Cg + nl : a.partial + size_t(t.split) * a.M * a.N + pcol + nl;
			const float sc = (GLU || fin) && live ? scg[nl] : 1.0f;
			const uint32_t acc = tmem_base + (uint32_t(quad * 32) << 16) + uint32_t(it & 1) * 256;
			const float4 *rs = reinterpret_cast<const float4 *>(a.rowscale + t.g0 * 8);
			// one token group: 32 accumulator columns = 4 digits x 8 tokens, and its row scales; lane i of the first eight: the largest
			// value recorded for token i so far (top1)
			auto request = [&](int g, uint32_t (&r)[32], float4 (&q)[2], uint32_t &seen) {
				tc_ld32(acc + uint32_t(g * 32), r);
				if (TOP1) seen = reinterpret_cast<const volatile uint32_t *>(a.top1)[2 * min((t.g0 + g) * 8 + (lane & 7), a.M - 1) + 1];
				q[0] = rs[2 * g];
				q[1] = rs[2 * g + 1];
			};
			auto finish = [&](int g, uint32_t (&r)[32], float4 (&q)[2], uint32_t seen, auto keep) {
				const int tok = (t.g0 + g) * 8;
				const float rsv[8] = {q[0].x, q[0].y, q[0].z, q[0].w, q[1].x, q[1].y, q[1].z, q[1].w};
				float v[8];
#pragma unroll
				for (int i = 0; i < 8; i++) {
					float y = float(int(r[24 + i]));
					y = fmaf(y, 256.0f, float(int(r[16 + i])));
					y = fmaf(y, 256.0f, float(int(r[8 + i])));
					y = fmaf(y, 256.0f, float(int(r[i])));
					v[i] = (y * rsv[i]) * sc;
				}
				if constexpr (GLU) {
					if (t.grp == 0) {
#pragma unroll
						for (int i = 0; i < 8; i++) kept[keep() + i] = v[i];
						return;
					}
					// GeluLut::index, eight at a time and selected instead of branched on (int(x) >= 0 is x > -1)
					float x[8], y[8];
					if (lut.inv != 0.0f) {
#pragma unroll
						for (int i = 0; i < 8; i++) x[i] = fmaf(v[i], lut.inv, lut_base);
					} else {
#pragma unroll
						for (int i = 0; i < 8; i++) x[i] = (v[i] - lut.mn) / lut.eps;
					}
#pragma unroll
					for (int i = 0; i < 8; i++) y[i] = lut_values[min(max(int(x[i]), 0), lut.size - 1)];
#pragma unroll
					for (int i = 0; i < 8; i++) {
						const float in = int(x[i]) < lut.size ? y[i] : v[i];
						v[i] = (x[i] > -1.0f && x[i] < 2147483648.0f ? in : 0.0f) * kept[keep() + i];
					}
				} else if constexpr (TOP1) {
					// Per token the largest value over the warp's 32 columns, the lowest column on equal values; NaN and -inf
					// never win. Lane i keeps token i's; only a key above the recorded one goes to the atomic. After a row's first
					// tiles hardly any value reaches what is recorded, and one vote says so (eight maxima over the lanes and a round
					// trip for the recorded keys each time made 256 rows of 1152 x 262144 slower than
					// writing them out and searching them by 15 us; with the vote it is 45 us faster).
					bool reaches = false;
#pragma unroll
					for (int i = 0; i < 8; i++) {
						const uint32_t b = __float_as_uint(v[i] + 0.0f);  // (-0 and +0 are equal)
						reaches |= (b ^ (uint32_t(int(b) >> 31) | 0x80000000u)) >= __shfl_sync(0xffffffffu, seen, i);
					}
					if (!__any_sync(0xffffffffu, reaches)) return;
					unsigned long long key = 0ull;
#pragma unroll
					for (int i = 0; i < 8; i++) {
						const uint32_t b = __float_as_uint(v[i] + 0.0f);  // (-0 and +0 are equal)
						const uint32_t ord = (v[i] > -INFINITY) ? ((b & 0x80000000u) ? ~b : (b | 0x80000000u)) : 0u;
						const uint32_t m = warp_umax(ord);
						const int src = __ffs(__ballot_sync(0xffffffffu, ord == m)) - 1;
						if (lane == i && m)
							key = (static_cast<unsigned long long>(m) << 32) | (0xFFFFFFFFu - uint32_t(a.top1_col0 + t.n0 + 128 * rank + quad * 32 + src));
					}
					if (lane < 8 && tok + lane < a.M && key > *reinterpret_cast<volatile unsigned long long *>(a.top1 + tok + lane))
						atomicMax(a.top1 + tok + lane, key);
					return;
				}
				float *p = dst + size_t(tok) * ld;
				if (tok + 8 <= a.M) {
#pragma unroll
					for (int i = 0; i < 8; i++, p += ld) *p = v[i];
				} else {
#pragma unroll
					for (int i = 0; i < 7; i++, p += ld)
						if (tok + i < a.M) *p = v[i];
				}
			};
			if (!tc_wait(&acc_full[it & 1], (it >> 1) & 1, a.err)) { s_fail = 1; break; }
			tc_fence_after();
			uint32_t ra[32], rb[32], sa = 0, sb = 0;
			float4 qa[2], qb[2];
			const int ng = live ? t.ng : 0;
			if (sub < ng) request(sub, ra, qa, sa);
			auto pair_of_groups = [&](int g, auto keep_a, auto keep_b) {
				asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
				if (g + 2 < ng) request(g + 2, rb, qb, sb);
				finish(g, ra, qa, sa, keep_a);
				if (g + 2 < ng) {
					asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
					if (g + 4 < ng) request(g + 4, ra, qa, sa);
					finish(g + 2, rb, qb, sb, keep_b);
				}
			};
			if constexpr (GLU) {  // (written out: what is kept is indexed by constants and stays in registers but for 24 bytes, at the limit of 168)
				static_assert(I8_TG == 8, "two pairs of token groups per warp");
				if (sub < ng) pair_of_groups(sub, [] { return 0; }, [] { return 8; });
				if (sub + 4 < ng) pair_of_groups(sub + 4, [] { return 16; }, [] { return 24; });
			} else {
#pragma unroll 1
				for (int g = sub; g < ng; g += 4) pair_of_groups(g, [] { return 0; }, [] { return 0; });
			}
			tc_fence_before();
			__syncwarp();
			if (lane == 0) {
				if (CG == 1 || rank == 0)
					mbar_arrive(&acc_free[it & 1]);
				else
					asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(i8_leader(&acc_free[it & 1])) : "memory");
			}
		}
	}
	// ---------------------------------------------------------------- teardown
	tc_fence_before();
	__syncthreads();
	if (warp == 0 && lane == 0 && rank == 0 && *(volatile int *)&s_fail) {
		// a wait ran out: every load that was issued must land before the shared memory is given up
		const int n = *(volatile int *)&s_issued;
		for (int c = max(0, n - NST); c < n; c++) {
			int spins = 0;
			while (!mbar_try_wait(&full_bar[c % NST], (c / NST) & 1) && ++spins < TC_SPIN_CAP) {
			}
		}
	}
	if (warp == 1 && rank == 0) {
		if (*(volatile int *)&s_fail && lane == 0) {  // let the MMAs in flight finish before the TMEM goes away
			int spins = 0;
			while (!mbar_try_wait(&drain_bar, 0) && ++spins < TC_SPIN_CAP) {
			}
		}
		__syncwarp();
	}
	if constexpr (CG == 2) {
		__syncthreads();
		i8_cluster_sync();  // neither CTA's memory is in use by the other any more
	}
	if (warp == 1) {
		tc_fence_after();
		if constexpr (CG == 1)
			asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
		else
			asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
	}
	if constexpr (CG == 2) {
		__syncthreads();
		i8_cluster_sync();
	}
}

}  // namespace tg
