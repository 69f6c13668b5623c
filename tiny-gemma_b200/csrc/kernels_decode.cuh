// Decode-step kernels (one token per sequence): embedding, the int8
// weight-only matvec with fused norm prologues / GeGLU epilogue, and split-KV
// attention over the cache. All are HBM-bandwidth bound; none uses tensor cores.
#pragma once
#include <cooperative_groups.h>

#include "tg_common.cuh"

namespace tg {

// =========================================================== embedding
// ops::embedding_decode, reference ops.hpp:574-616:
//   h[d] = scale[d] * (sqrt(D) * float(wte[tok, d]))
// One CTA per sequence. Also latches the position this step works at:
// step_pos = next_pos, next_pos += 1 (KVCache::position_ptr, decode.hpp:69).
struct EmbedArgs {
	const int8_t *wte;
	const float *scales;
	const int *tok;   // [B]
	float *h;         // [B][D]
	int *step_pos;    // [B]
	int *next_pos;    // [B]
	int *err_flag;    // set to 1 if a token id is out of range
	int D, V;
	float sqrtD;
};

__global__ void embed_decode_kernel(EmbedArgs a) {
	pdl_trigger();
	pdl_wait();
	int b = blockIdx.x;
	int tok = a.tok[b];
	if (tok < 0 || tok >= a.V) {
		if (threadIdx.x == 0) *a.err_flag = 1;
		tok = 0;
	}
	const int8_t *row = a.wte + size_t(tok) * a.D;
	for (int d = threadIdx.x; d < a.D; d += blockDim.x) a.h[size_t(b) * a.D + d] = a.scales[d] * (a.sqrtD * float(row[d]));
	if (threadIdx.x == 0) {
		int p = a.next_pos[b];
		a.step_pos[b] = p;
		a.next_pos[b] = p + 1;
	}
}

// =========================================================== int8 matvec
// y[n] = scale[n] * sum_k x[k] * W[k,n]   (gemv::qgemv, reference linalg.hpp:41-108)
//
// W is [K,N] row-major int8 exactly as in gemma_i8.bin, so consecutive columns
// are consecutive bytes: a lane owns 16 columns (one 128-bit load per row), 8
// lanes cover a 128-column tile and the 4 lane groups of a warp take 4
// different rows, so one warp-wide load instruction fetches four full 128-byte
// lines. A CTA (8 warps) walks 32 rows per iteration over its K-chunk.
//
// Small-N matrices are split along K across CTAs (grid.y); partial sums go to
// a scratch array and the last CTA to finish a column tile (ticket counter)
// adds them in split order — deterministic, no floating-point atomics.
//
// Prologues build the CTA's slice of x in shared memory:
//   PRO_PLAIN    x = in
//   PRO_NORM     x = rmsnorm(h; w_pre)
//   PRO_RESNORM  h' = h + rmsnorm(t; w_post);  x = rmsnorm(h'; w_pre)   (CTA 0,0 stores h')
//   (modules::attention / modules::mlp sandwich norms, reference modules.hpp:140,166-168,209,218-219)
// Epilogues (by the finishing CTA of a tile):
//   EPI_SCALE    out = scale * sum
//   EPI_GEGLU    two matrices (up, gate) share the tile: out = lut(sg*gate) * (su*up)
//   (ops::gelu + ops::mul, reference modules.hpp:213-215)
constexpr int MV_TN = 128;
constexpr int MV_THREADS = 256;
constexpr int MV_NWARPS = MV_THREADS / 32;
constexpr int MV_ROWS_PER_ITER = 32;

enum { PRO_PLAIN = 0, PRO_NORM = 1, PRO_RESNORM = 2 };
enum { EPI_SCALE = 0, EPI_GEGLU = 1 };

struct MvSeg {
	const int8_t *w;
	const float *scale;
	int N;        // row stride of this matrix
	int out_off;  // column offset of this segment in the output row
	int tile0;    // first tile index of this segment
};

struct MvArgs {
	MvSeg seg[3];
	int nseg;
	int ntiles;      // total column tiles over all segments (EPI_GEGLU: tiles of one matrix)
	int K;           // rows
	int kc;          // rows per K-split (multiple of 32)
	int nsplit;      // == gridDim.y
	int B;           // sequences in this launch (<= MB)
	int part_stride; // columns per (split, b) row of the partial buffer
	int out_stride;  // floats per output row
	// prologue inputs
	const float *x;       // PRO_PLAIN: [B][K]
	const float *h;       // PRO_NORM / PRO_RESNORM: residual stream [B][K]
	const float *t;       // PRO_RESNORM: branch output to be post-normed [B][K]
	const float *w_post;  // [K]
	const float *w_pre;   // [K]
	float *h_out;         // PRO_RESNORM: updated residual stream [B][K] (must differ from h)
	float *x_out;         // optional copy of the normed input (parity read-back), may be null
	// split-K machinery
	float *partial;       // [nsplit][B][part_stride]
	unsigned *tickets;    // [ntiles], zero on entry, zero on exit
	float *out;           // [B][out_stride]
	GeluLut lut;          // EPI_GEGLU
};

template <int MB>
__device__ __forceinline__ void mv_accumulate(float (&acc)[MB][16], const int4 &v, const float (&xv)[MB]) {
	const uint32_t words[4] = {uint32_t(v.x), uint32_t(v.y), uint32_t(v.z), uint32_t(v.w)};
#pragma unroll
	for (int j = 0; j < 4; j++) {
		float f[4];
		i8x4_to_f32(words[j], f);
#pragma unroll
		for (int b = 0; b < MB; b++) {
#pragma unroll
			for (int i = 0; i < 4; i++) acc[b][4 * j + i] = fmaf(xv[b], f[i], acc[b][4 * j + i]);
		}
	}
}

// Walks rows [k0, k0+kc) of one 128-column tile; returns per-thread sums for
// its 16 columns over the rows this thread visited.
template <int MB>
__device__ __forceinline__ void mv_tile_rows(float (&acc)[MB][16], const int8_t *wcol, int N, int kc, const float *xs,
                                             int xs_stride) {
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int sub = lane >> 3;
	const int r0 = warp * 4 + sub;  // row within a 32-row iteration
	const int8_t *p = wcol + size_t(r0) * N;
	const size_t step = size_t(MV_ROWS_PER_ITER) * N;
	const int iters = kc / MV_ROWS_PER_ITER;
	int it = 0;
	// eight 16-byte loads in flight per thread (32 KB per CTA): a K-split slice of 256 rows is one round trip to DRAM
	for (; it + 8 <= iters; it += 8) {
		int4 v[8];
#pragma unroll
		for (int u = 0; u < 8; u++) v[u] = ld_stream_int4(p + u * step);
		p += 8 * step;
		const int r = it * MV_ROWS_PER_ITER + r0;
#pragma unroll
		for (int u = 0; u < 8; u++) {
			float xv[MB];
#pragma unroll
			for (int b = 0; b < MB; b++) xv[b] = xs[b * xs_stride + r + 32 * u];
			mv_accumulate<MB>(acc, v[u], xv);
		}
	}
	for (; it + 4 <= iters; it += 4) {
		int4 v0 = ld_stream_int4(p);
		int4 v1 = ld_stream_int4(p + step);
		int4 v2 = ld_stream_int4(p + 2 * step);
		int4 v3 = ld_stream_int4(p + 3 * step);
		p += 4 * step;
		float xv[MB];
		const int r = it * MV_ROWS_PER_ITER + r0;
#pragma unroll
		for (int b = 0; b < MB; b++) xv[b] = xs[b * xs_stride + r];
		mv_accumulate<MB>(acc, v0, xv);
#pragma unroll
		for (int b = 0; b < MB; b++) xv[b] = xs[b * xs_stride + r + 32];
		mv_accumulate<MB>(acc, v1, xv);
#pragma unroll
		for (int b = 0; b < MB; b++) xv[b] = xs[b * xs_stride + r + 64];
		mv_accumulate<MB>(acc, v2, xv);
#pragma unroll
		for (int b = 0; b < MB; b++) xv[b] = xs[b * xs_stride + r + 96];
		mv_accumulate<MB>(acc, v3, xv);
	}
	for (; it < iters; it++) {
		int4 v0 = ld_stream_int4(p);
		p += step;
		float xv[MB];
		const int r = it * MV_ROWS_PER_ITER + r0;
#pragma unroll
		for (int b = 0; b < MB; b++) xv[b] = xs[b * xs_stride + r];
		mv_accumulate<MB>(acc, v0, xv);
	}
}

// Reduce the per-thread sums of one tile across the CTA: over the 4 row groups
// of each warp by shuffle, then over the 8 warps through shared memory.
// On return threads 0..127 hold, for each b, the tile's column (threadIdx.x).
template <int MB>
__device__ __forceinline__ void mv_reduce_cta(float (&acc)[MB][16], float *red /*[MB][NWARPS][128]*/, float (&col)[MB]) {
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
	for (int b = 0; b < MB; b++)
#pragma unroll
		for (int i = 0; i < 16; i++) {
			float v = acc[b][i];
			v += __shfl_xor_sync(0xffffffffu, v, 8);
			v += __shfl_xor_sync(0xffffffffu, v, 16);
			acc[b][i] = v;
		}
	__syncthreads();
	if (lane < 8) {
#pragma unroll
		for (int b = 0; b < MB; b++)
#pragma unroll
			for (int i = 0; i < 16; i++) red[(b * MV_NWARPS + warp) * MV_TN + lane * 16 + i] = acc[b][i];
	}
	__syncthreads();
	if (threadIdx.x < MV_TN) {
#pragma unroll
		for (int b = 0; b < MB; b++) {
			float s = 0.0f;
#pragma unroll
			for (int w = 0; w < MV_NWARPS; w++) s += red[(b * MV_NWARPS + w) * MV_TN + threadIdx.x];
			col[b] = s;
		}
	}
}

template <int MB, int PRO, int EPI>
__global__ void __launch_bounds__(MV_THREADS) qmatvec_kernel(MvArgs a) {
	extern __shared__ float smem[];
	// layout: xs[MB][kc] | hs[MB][K] (norm prologues only) | red[MB][8][128] (x2 for GEGLU) | misc
	float *xs = smem;
	float *hs = xs + MB * a.kc;
	float *red = hs + ((PRO == PRO_PLAIN) ? 0 : MB * a.K);
	float *red2 = red + MB * MV_NWARPS * MV_TN;
	__shared__ float bred[MV_NWARPS];
	__shared__ int s_last;

	const int split = blockIdx.y;
	const int k0 = split * a.kc;
	const int tid = threadIdx.x;

	// ------------------------------------------------------------ prologue
	if (PRO == PRO_PLAIN) {
		for (int b = 0; b < a.B; b++)
			for (int k = tid; k < a.kc; k += MV_THREADS) xs[b * a.kc + k] = a.x[size_t(b) * a.K + k0 + k];
	} else {
		const int D = a.K;
		for (int b = 0; b < a.B; b++) {
			float *hb = hs + b * D;
			if (PRO == PRO_RESNORM) {
				float ss = 0.0f;
				for (int d = tid; d < D; d += MV_THREADS) {
					float v = a.t[size_t(b) * D + d];
					ss = fmaf(v, v, ss);
				}
				ss = block_sum<MV_NWARPS>(ss, bred);
				const float r1 = inv_rms(ss, D);
				for (int d = tid; d < D; d += MV_THREADS) {
					float v = a.t[size_t(b) * D + d];
					hb[d] = a.h[size_t(b) * D + d] + (v * r1) * (a.w_post[d] + 1.0f);
				}
			} else {
				for (int d = tid; d < D; d += MV_THREADS) hb[d] = a.h[size_t(b) * D + d];
			}
			float ss2 = 0.0f;
			for (int d = tid; d < D; d += MV_THREADS) {
				float v = hb[d];
				ss2 = fmaf(v, v, ss2);
			}
			ss2 = block_sum<MV_NWARPS>(ss2, bred);
			const float r2 = inv_rms(ss2, D);
			for (int k = tid; k < a.kc; k += MV_THREADS) xs[b * a.kc + k] = (hb[k0 + k] * r2) * (a.w_pre[k0 + k] + 1.0f);
			if (blockIdx.x == 0 && blockIdx.y == 0) {
				if (PRO == PRO_RESNORM)
					for (int d = tid; d < D; d += MV_THREADS) a.h_out[size_t(b) * D + d] = hb[d];
				if (a.x_out)
					for (int d = tid; d < D; d += MV_THREADS) a.x_out[size_t(b) * D + d] = (hb[d] * r2) * (a.w_pre[d] + 1.0f);
			}
		}
	}
	for (int b = a.B; b < MB; b++)
		for (int k = tid; k < a.kc; k += MV_THREADS) xs[b * a.kc + k] = 0.0f;
	__syncthreads();

	const int lane = tid & 31;
	const int cg = lane & 7;  // 16-column group inside the tile

	// ------------------------------------------------------------ tiles
	for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x) {
		// locate the segment of this tile
		int sidx = 0;
		if (EPI != EPI_GEGLU) {
			while (sidx + 1 < a.nseg && tile >= a.seg[sidx + 1].tile0) sidx++;
		}
		const MvSeg &sg = a.seg[sidx];
		const int n0 = (tile - sg.tile0) * MV_TN;  // first column of the tile inside its matrix

		float acc[MB][16];
#pragma unroll
		for (int b = 0; b < MB; b++)
#pragma unroll
			for (int i = 0; i < 16; i++) acc[b][i] = 0.0f;
		mv_tile_rows<MB>(acc, sg.w + size_t(k0) * sg.N + n0 + cg * 16, sg.N, a.kc, xs, a.kc);
		float col[MB];
		mv_reduce_cta<MB>(acc, red, col);

		float col2[MB];
		if (EPI == EPI_GEGLU) {
			const MvSeg &gg = a.seg[1];
#pragma unroll
			for (int b = 0; b < MB; b++)
#pragma unroll
				for (int i = 0; i < 16; i++) acc[b][i] = 0.0f;
			mv_tile_rows<MB>(acc, gg.w + size_t(k0) * gg.N + n0 + cg * 16, gg.N, a.kc, xs, a.kc);
			mv_reduce_cta<MB>(acc, red2, col2);
		}

		const int pcol = sg.out_off + n0 + tid;  // column in the partial / plain output row
		if (a.nsplit == 1) {
			if (tid < MV_TN) {
				for (int b = 0; b < a.B; b++) {
					if (EPI == EPI_SCALE) {
						a.out[size_t(b) * a.out_stride + pcol] = col[b] * sg.scale[n0 + tid];
					} else {
						float up = col[b] * sg.scale[n0 + tid];
						float gate = col2[b] * a.seg[1].scale[n0 + tid];
						a.out[size_t(b) * a.out_stride + n0 + tid] = a.lut(gate) * up;
					}
				}
			}
			continue;
		}

		// split-K: publish partials, take a ticket, last CTA of the tile finishes
		if (tid < MV_TN) {
			for (int b = 0; b < a.B; b++) {
				float *prow = a.partial + (size_t(split) * a.B + b) * a.part_stride;
				if (EPI == EPI_SCALE) {
					__stcg(prow + pcol, col[b]);
				} else {
					__stcg(prow + n0 + tid, col[b]);
					__stcg(prow + a.seg[1].out_off + n0 + tid, col2[b]);
				}
			}
		}
		__threadfence();
		__syncthreads();
		if (tid == 0) {
			unsigned tk = atomicAdd(&a.tickets[tile], 1u);
			s_last = (tk == unsigned(a.nsplit - 1));
		}
		__syncthreads();
		if (s_last) {
			__threadfence();
			if (tid < MV_TN) {
				for (int b = 0; b < a.B; b++) {
					// the splits are added in ascending order, eight loads in flight at a time (a chain of
					// dependent loads over 30 splits cost more than the matvec itself)
					float s1 = 0.0f, s2 = 0.0f;
					const float *prow0 = a.partial + size_t(b) * a.part_stride;
					const size_t sstride = size_t(a.B) * a.part_stride;
					if (EPI == EPI_SCALE) {
						s1 = sum_splits<true>(prow0 + pcol, sstride, a.nsplit);
					} else {
						s1 = sum_splits<true>(prow0 + n0 + tid, sstride, a.nsplit);
						s2 = sum_splits<true>(prow0 + a.seg[1].out_off + n0 + tid, sstride, a.nsplit);
					}
					if (EPI == EPI_SCALE) {
						a.out[size_t(b) * a.out_stride + pcol] = s1 * sg.scale[n0 + tid];
					} else {
						float up = s1 * sg.scale[n0 + tid];
						float gate = s2 * a.seg[1].scale[n0 + tid];
						a.out[size_t(b) * a.out_stride + n0 + tid] = a.lut(gate) * up;
					}
				}
			}
			if (tid == 0) a.tickets[tile] = 0u;
		}
		__syncthreads();
	}
}

// =========================================================== single-wave matvec (one sequence)
// y[n] = scale[n] * sum_k x[k] W[k,n] for matrices small enough that one wave of CTAs holds all of W in
// flight at once (the layer matrices: 0.6 - 8 MB). Such a launch is bound by its chain of dependent memory
// round trips, so there is exactly one: every CTA requests its whole K-slice of a column tile (and its
// x values) before it waits for anything. K is split over the CTAs of a thread-block cluster
// (gridDim.y = cluster size <= 8) whose partial sums meet in the shared memory of the cluster's first CTA
// (distributed shared memory), added in rank order: no partial-sum buffer, no tickets, no second launch,
// the same bits on every run.
// A column tile is 16 * TPR columns (TPR = 1, 2, 4 threads per row, 16 int8 each); thread t takes columns
// 16 * (t % TPR) .. of rows t / TPR, t / TPR + threads / TPR, ...; at most MVC_MAX_IT rows per thread
// (512 or 256 threads per CTA).
constexpr int MVC_MAX_IT = 10;
constexpr int MVC_MAX_CLUSTER = 8;

template <int TPR, int MVC_THREADS>
__global__ void __launch_bounds__(MVC_THREADS, 1) qmatvec_cluster_kernel(float *y, const float *x, const int8_t *w, const float *scales,
                                                                         int K, int N, int kc) {
	namespace cg = cooperative_groups;
	constexpr int TN = 16 * TPR, ROWS = MVC_THREADS / TPR, MVC_NWARPS = MVC_THREADS / 32;
	cg::cluster_group cluster = cg::this_cluster();
	pdl_trigger();
	pdl_wait();
	__shared__ __align__(16) float red[MVC_NWARPS][TN];
	__shared__ float part[MVC_MAX_CLUSTER][TN];  // (used in the cluster's first CTA)
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int n0 = blockIdx.x * TN;
	const int rank = int(cluster.block_rank()), nranks = int(cluster.num_blocks());
	const int k0 = rank * kc;
	const int r0 = tid / TPR, cgp = tid % TPR;
	const int8_t *p = w + size_t(k0 + r0) * N + n0 + cgp * 16;
	int4 v[MVC_MAX_IT];
	float xv[MVC_MAX_IT];
#pragma unroll
	for (int it = 0; it < MVC_MAX_IT; it++) {
		const int r = r0 + it * ROWS;
		v[it] = make_int4(0, 0, 0, 0);
		xv[it] = 0.0f;
		if (r < kc) {
			v[it] = ld_stream_int4(p + size_t(it) * ROWS * N);
			xv[it] = __ldg(x + k0 + r);
		}
	}
	float sc = 0.0f;
	if (rank == 0 && tid < TN) sc = __ldg(scales + n0 + tid);
	float acc[16];
#pragma unroll
	for (int i = 0; i < 16; i++) acc[i] = 0.0f;
#pragma unroll
	for (int it = 0; it < MVC_MAX_IT; it++) {
		const uint32_t words[4] = {uint32_t(v[it].x), uint32_t(v[it].y), uint32_t(v[it].z), uint32_t(v[it].w)};
#pragma unroll
		for (int j = 0; j < 4; j++) {
			float f[4];
			i8x4_to_f32(words[j], f);
#pragma unroll
			for (int i = 0; i < 4; i++) acc[4 * j + i] = fmaf(xv[it], f[i], acc[4 * j + i]);
		}
	}
	// over the rows of a warp (lanes with the same column group), then over the warps
#pragma unroll
	for (int i = 0; i < 16; i++) {
		float s = acc[i];
#pragma unroll
		for (int o = TPR; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
		acc[i] = s;
	}
	if (lane < TPR) {
#pragma unroll
		for (int i = 0; i < 16; i += 4)
			*reinterpret_cast<float4 *>(&red[warp][lane * 16 + i]) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
	}
	__syncthreads();
	if (tid < TN) {
		float s = 0.0f;
#pragma unroll
		for (int wi = 0; wi < MVC_NWARPS; wi++) s += red[wi][tid];
		float *dst = cluster.map_shared_rank(&part[rank][tid], 0);  // this rank's row in the first CTA's array
		*dst = s;
	}
	cluster.sync();  // (every thread of every CTA: the stores above are visible to the first CTA behind it)
	if (rank == 0 && tid < TN) {
		float s = 0.0f;
		for (int r = 0; r < nranks; r++) s += part[r][tid];
		y[n0 + tid] = s * sc;
	}
}

// =========================================================== wide matvec (one sequence, the vocabulary matrix)
// y[n] = scale[n] * sum_k x[k] W[k,n] for a matrix of hundreds of MB: HBM bound. One CTA per SM owns `groups` groups of
// 16 consecutive columns (262144 columns over 148 SMs: 112 groups, 1792 contiguous bytes of every row, whole lines) in
// four row sets. A thread copies its own 16-byte pieces into a ring of stages of eight rows in shared memory (cp.async, no
// barrier: it reads nobody else's) and works on one stage with the next on their way, 57 KB each per SM.
// KEPT, a matrix that the L2 holds (of the accepted depths 256, 67 MB): three stages; such a launch is mostly its own start, and the next call finds
// lines of it. Otherwise two stages, evict-first in the L2: nothing is read twice, and at normal priority the reads push out the dirty lines that
// earlier kernels left there, whose way to DRAM then goes with them (126 MB behind a kernel that wrote as much: a third of the launch).
// In us, several matrices in turn / one again after a pause / the same after 400 MB were written:
//                                  256 x 262144            640 x 262144            1152 x 262144           2048 x 262144
//     loads into registers         17.3 / 22.4 / 29.1      34.4 / 41.8 / 44.5      56.2 / 62.9 / 67.6      95.1 / 104 / 112
//     3 stages, normal priority    17.1 / 20.6 / 29.2 (*)  33.5 / 39.8 / 49.0      54.8 / 60.3 / 75.4      92.7 / 99.7 / 117
//     3 stages, evict-first        15.7 / 21.0 / 28.0      32.9 / 37.2 / 42.7      54.3 / 59.2 / 66.1      92.1 / 96.2 / 107
//     2 stages, normal priority    20.4 / 20.7 / 29.0      31.6 / 38.0 / 46.2      50.7 / 56.8 / 71.9      83.5 / 90.6 / 112
//     2 stages, evict-first        18.8 / 20.5 / 27.0      30.7 / 37.8 / 42.8      50.0 / 55.2 / 61.6      83.5 / 89.1 / 99.5
// (*) 13.1 for one matrix back to back (evict-first 15.2). 50.0 us are 6.0 TB/s. First pass over 302 MB that were just made: 67, 77, 63 and, with two stages
// evict-first, 60. Groups of 111, whose pieces of a row begin anywhere in a line, took 59.9 where 112 took 54.9; single FMAs instead of paired ones
// 52.0 instead of 50.4.
constexpr int MVW_SETS = 4, MVW_MAX_GROUPS = 128, MVW_U = 8;
__host__ __device__ constexpr int mvw_stages(bool kept) { return kept ? 3 : 2; }
template <bool KEPT>
__device__ __forceinline__ void mvw_copy(uint32_t dst, const int8_t *src, uint64_t policy) {
	if constexpr (KEPT)
		asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
	else
		asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "l"(policy) : "memory");
}
// a += (b - (2^23 + 128)) * c, both halves: b holds the bits of 2^23 + 128 + a weight (exact, see i8_lane_to_f32)
__device__ __forceinline__ void mvw_fma2(float2 &a, uint32_t b0, uint32_t b1, float c) {
	asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tmov.b64 z, {%5, %5};\n\t"
	    "add.rn.f32x2 y, y, z;\n\tmov.b64 z, {%4, %4};\n\tfma.rn.f32x2 x, y, z, x;\n\tmov.b64 {%0, %1}, x;\n\t}"
	    : "+f"(a.x), "+f"(a.y)
	    : "r"(b0), "r"(b1), "f"(c), "f"(-8388736.0f));
}
template <bool KEPT>
__global__ void __launch_bounds__(MVW_SETS *MVW_MAX_GROUPS, 1) qmatvec_wide_kernel(float *y, const float *x, const int8_t *w, const float *scales,
                                                                                   int K, int N, int groups) {
	extern __shared__ __align__(16) float mvw_smem[];  // x [K], the ring [stages][8][threads] of 16 bytes; the row sets' sums [4][groups * 16] in its place
	pdl_trigger();
	pdl_wait();
	float *xs = mvw_smem;
	const int tid = threadIdx.x, nt = blockDim.x;
	const int set = tid / groups, g = tid - set * groups;
	const int col = (blockIdx.x * groups + g) * 16;
	const bool on = set < MVW_SETS && col < N;
	const int8_t *p = w + size_t(on ? set : 0) * N + (on ? col : 0);
	const size_t step = size_t(MVW_SETS) * N;
	const int n = on ? K / MVW_SETS : 0;  // K is a multiple of 4 * MVW_U
	const uint32_t ring = uint32_t(__cvta_generic_to_shared(xs + K)) + 16u * tid;
	constexpr int STAGES = mvw_stages(KEPT);
	uint64_t policy = 0;
	if constexpr (!KEPT) asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
	int next = 0;  // rows requested so far
	auto request = [&](int st) {
		if (next < n) {
#pragma unroll
			for (int u = 0; u < MVW_U; u++) mvw_copy<KEPT>(ring + uint32_t((st * MVW_U + u) * nt) * 16u, p + u * step, policy);
			p += MVW_U * step;
			next += MVW_U;
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
#pragma unroll
	for (int st = 0; st < STAGES; st++) request(st);
	for (int k = tid; k < K; k += nt) xs[k] = x[k];
	__syncthreads();
	float2 acc[8];
#pragma unroll
	for (int i = 0; i < 8; i++) acc[i] = make_float2(0.0f, 0.0f);
	int st = 0;
#pragma unroll 1
	for (int it = 0; it < n; it += MVW_U) {
		asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
#pragma unroll
		for (int u = 0; u < MVW_U; u++) {
			uint32_t words[4];
			asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
			             : "=r"(words[0]), "=r"(words[1]), "=r"(words[2]), "=r"(words[3])
			             : "r"(ring + uint32_t((st * MVW_U + u) * nt) * 16u)
			             : "memory");
			const float xv = xs[(it + u) * MVW_SETS + set];
#pragma unroll
			for (int j = 0; j < 4; j++) {
				const uint32_t b = words[j] ^ 0x80808080u;  // (as i8x4_to_f32)
				mvw_fma2(acc[2 * j], __byte_perm(b, 0x4B000000u, 0x7650u), __byte_perm(b, 0x4B000000u, 0x7651u), xv);
				mvw_fma2(acc[2 * j + 1], __byte_perm(b, 0x4B000000u, 0x7652u), __byte_perm(b, 0x4B000000u, 0x7653u), xv);
			}
		}
		request(st);
		if (++st == STAGES) st = 0;
	}
	asm volatile("cp.async.wait_group 0;" ::: "memory");
	__syncthreads();  // (the ring is done with everywhere)
	float *sums = xs + K;
	if (set < MVW_SETS) {
#pragma unroll
		for (int i = 0; i < 8; i += 2)
			*reinterpret_cast<float4 *>(sums + (set * groups + g) * 16 + 2 * i) = make_float4(acc[i].x, acc[i].y, acc[i + 1].x, acc[i + 1].y);
	}
	__syncthreads();
	for (int c = tid; c < groups * 16; c += nt) {
		const int cn = blockIdx.x * groups * 16 + c;
		if (cn >= N) break;
		float s = 0.0f;
#pragma unroll
		for (int r = 0; r < MVW_SETS; r++) s += sums[r * groups * 16 + c];
		y[cn] = s * scales[cn];
	}
}

// =========================================================== final hidden state
// x = rmsnorm(h + rmsnorm(t; w_post); w_final) per sequence — the prologue of
// the lm_head (reference modules.hpp:242-246) as a kernel of its own, for callers
// that score the vocabulary elsewhere (vocab-sharded lm_head). One CTA per sequence.
__global__ void __launch_bounds__(256) final_hidden_kernel(float *x_out, const float *h, const float *t, const float *w_post,
                                                           const float *w_final, int D) {
	__shared__ float bred[8];
	extern __shared__ float hs[];
	const int b = blockIdx.x, tid = threadIdx.x;
	float ss = 0.0f;
	for (int d = tid; d < D; d += 256) {
		float v = t[size_t(b) * D + d];
		ss = fmaf(v, v, ss);
	}
	ss = block_sum<8>(ss, bred);
	const float r1 = inv_rms(ss, D);
	float ss2 = 0.0f;
	for (int d = tid; d < D; d += 256) {
		float v = h[size_t(b) * D + d] + (t[size_t(b) * D + d] * r1) * (w_post[d] + 1.0f);
		hs[d] = v;
		ss2 = fmaf(v, v, ss2);
	}
	ss2 = block_sum<8>(ss2, bred);
	const float r2 = inv_rms(ss2, D);
	for (int d = tid; d < D; d += 256) x_out[size_t(b) * D + d] = (hs[d] * r2) * (w_final[d] + 1.0f);
}

// =========================================================== attention (decode)
// Per sequence and layer: q/k RMSNorm (per head), RoPE at the token's position,
// KV append into the (ring) cache, then one query against every valid cache
// slot for the 4 query heads that share the single KV head.
// (modules::attention decode branch, reference modules.hpp:151-159;
//  RoPE decode.hpp:136-211; KVCache::update_single decode.hpp:49-70;
//  ops::attention_decode ops.hpp:224-370.)
//
// (The batched kernel is attn_decode_kernel in kernels_attn_cc.cuh; here is what the persistent kernels share with it.)
constexpr int AT_HD = 256;
constexpr int AT_NH = 4;

__device__ __forceinline__ void norm_rope_head(const float *x, const float *w, const float *cosr, const float *sinr,
                                                float scale, float *dst) {
	// one warp; lane owns d = 4*lane..4*lane+3 and the partner 128 + the same
	const int lane = threadIdx.x & 31;
	float lo[4], hi[4];
	float ss = 0.0f;
#pragma unroll
	for (int i = 0; i < 4; i++) {
		lo[i] = x[4 * lane + i];
		hi[i] = x[128 + 4 * lane + i];
		ss = fmaf(lo[i], lo[i], ss);
		ss = fmaf(hi[i], hi[i], ss);
	}
	ss = warp_sum(ss);
	const float r = inv_rms(ss, AT_HD);
#pragma unroll
	for (int i = 0; i < 4; i++) {
		const int d = 4 * lane + i;
		float a = (lo[i] * r) * (w[d] + 1.0f);
		float b = (hi[i] * r) * (w[d + 128] + 1.0f);
		// y = cos*x + rotate_half(x)*sin, rotate_half = [-x_hi, x_lo]
		float ylo = fmaf(-1.0f * b, sinr[d], cosr[d] * a);
		float yhi = fmaf(a, sinr[d + 128], cosr[d + 128] * b);
		dst[d] = ylo * scale;
		dst[d + 128] = yhi * scale;
	}
}

}  // namespace tg
