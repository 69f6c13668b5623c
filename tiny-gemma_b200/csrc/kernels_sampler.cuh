// On-device samplers over the 262144-way logits row of each sequence.
#pragma once
#include "tg_common.cuh"

namespace tg {

struct SampleArgs {
	float *logits;   // [B][V]; min-p overwrites it with the reference's "probabilities"
	int V;
	int *tok_out;    // [B] token fed to the next decode step
	int *tok_log;    // [max_steps][B] or null
	int *log_count;  // [B] entries written so far per sequence (device counter)
	int log_cap;     // capacity in steps
	int B;
	// min-p
	float minp, temp;
	const float *randf;  // [n][B] uniforms, indexed by randf_count[b]
	int *randf_count;    // [B]
	int randf_cap;
};

__device__ __forceinline__ void emit_token(const SampleArgs &a, int b, int tok) {
	a.tok_out[b] = tok;
	if (a.tok_log) {
		int c = a.log_count[b];
		if (c < a.log_cap) a.tok_log[size_t(c) * a.B + b] = tok;
		a.log_count[b] = c + 1;
	}
}

// ops::argmax_logits, reference ops.hpp:744-760: ascending scan with a strict
// '>' — the lowest index wins ties, NaN never wins, -1 if nothing exceeds -inf.
// grid (V / SR_PART rounded up, rows): a row is 1 MB, which one CTA reads in ~35 us (a chain of dependent round trips)
// and 32 CTAs in ~3. The CTAs of a row meet in a 64-bit key (larger value first, then the lower index); the one that
// arrives last emits the token and leaves key and ticket zero for the next launch.
constexpr int SR_THREADS = 256;
constexpr int SR_PART = 8192;  // columns per CTA
__global__ void __launch_bounds__(SR_THREADS) argmax_kernel(SampleArgs a, unsigned long long *keys, unsigned *tickets) {
	pdl_trigger();
	pdl_wait();
	__shared__ unsigned long long sk[SR_THREADS / 32];
	const int b = blockIdx.y, tid = threadIdx.x;
	const float *x = a.logits + size_t(b) * a.V;
	float4 v[SR_PART / (4 * SR_THREADS)];
#pragma unroll
	for (int j = 0; j < SR_PART / (4 * SR_THREADS); j++) {
		const int i = blockIdx.x * SR_PART + 4 * (tid + SR_THREADS * j);
		v[j] = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
		if (i < a.V) v[j] = __ldcg(reinterpret_cast<const float4 *>(x + i));
	}
	float best = -INFINITY;
	int arg = -1;
#pragma unroll
	for (int j = 0; j < SR_PART / (4 * SR_THREADS); j++) {
		const int i = blockIdx.x * SR_PART + 4 * (tid + SR_THREADS * j);
		if (v[j].x > best) { best = v[j].x; arg = i; }
		if (v[j].y > best) { best = v[j].y; arg = i + 1; }
		if (v[j].z > best) { best = v[j].z; arg = i + 2; }
		if (v[j].w > best) { best = v[j].w; arg = i + 3; }
	}
	unsigned long long key = 0ull;
	if (arg >= 0) {
		const uint32_t u = __float_as_uint(best == 0.0f ? 0.0f : best);  // (-0 and +0 are equal)
		key = (static_cast<unsigned long long>((u & 0x80000000u) ? ~u : (u | 0x80000000u)) << 32) | (0xFFFFFFFFu - uint32_t(arg));
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) key = max(key, __shfl_xor_sync(0xffffffffu, key, o));
	if ((tid & 31) == 0) sk[tid >> 5] = key;
	__syncthreads();
	if (tid == 0) {
		for (int w = 1; w < SR_THREADS / 32; w++) key = max(key, sk[w]);
		if (key) atomicMax(keys + b, key);
		__threadfence();
		if (atomicAdd(tickets + b, 1u) == gridDim.x - 1) {
			__threadfence();
			const unsigned long long k = atomicExch(keys + b, 0ull);
			tickets[b] = 0u;
			emit_token(a, b, k ? int(0xFFFFFFFFu - uint32_t(k)) : -1);
		}
	}
}

// the tokens of the rows' keys that the vocabulary GEMM left (the same keys); they go back to zero for the next launch
__global__ void top1_emit_kernel(SampleArgs a, unsigned long long *keys) {
	pdl_trigger();
	pdl_wait();
	const int b = blockIdx.x * blockDim.x + threadIdx.x;
	if (b >= a.B) return;
	const unsigned long long k = keys[b];
	keys[b] = 0ull;
	emit_token(a, b, k ? int(0xFFFFFFFFu - uint32_t(k)) : -1);
}

// ------------------------------------------------------------------ exact parallel inverse CDF
// Step (6) of min-p sampling is "the first index whose running fp32 sum reaches randf", where the
// running sum is the sequential chain cum = fl(cum + p[i]). fp32 addition is not associative, so a
// tree sum would move the crossing index. The chain can still be evaluated in parallel, exactly:
// while cum stays in one binade [2^e, 2^(e+1)) it is an integer multiple S of u = 2^(e-23), and
// adding p rounds S + p/u to the nearest integer, ties to even. So element i acts on S as
//     S -> S + a0[i]  (S even),   S -> S + a1[i]  (S odd),
// with a0 = a1 = round(p/u) except on an exact tie, where the pair encodes round-half-even. Such
// maps compose into maps of the same form (the parity of the result follows from the parity of the
// input), so a prefix scan of (a0, a1) pairs gives every partial sum of the chain, bit for bit.
// A block in which the sum leaves the binade is added up element by element, and the maps go on behind
// it with the new u. Sums saturate far above every threshold, so they stay monotone.
struct CdfFn {
	int a0, a1;
};
constexpr int CDF_SAT = 1 << 27;
constexpr int CDF_BIG = 1 << 25;
__device__ __forceinline__ CdfFn cdf_compose(CdfFn f, CdfFn g) {  // first f, then g
	CdfFn h;
	h.a0 = min(CDF_SAT, f.a0 + ((f.a0 & 1) ? g.a1 : g.a0));
	h.a1 = min(CDF_SAT, f.a1 + ((f.a1 & 1) ? g.a0 : g.a1));
	return h;
}
__device__ __forceinline__ int cdf_apply(CdfFn f, int S) { return min(CDF_SAT, S + ((S & 1) ? f.a1 : f.a0)); }
__device__ __forceinline__ CdfFn cdf_element(float p, float inv_u) {
	const float x = p * inv_u;
	CdfFn f;
	if (!(x < 33554432.0f)) {  // also NaN / inf: forces the fp32 path for this element
		f.a0 = f.a1 = CDF_BIG;
		return f;
	}
	const float fl = floorf(x);
	const float fr = x - fl;  // exact
	const int q = int(fl);
	if (fr == 0.5f) {
		f.a0 = q + (q & 1);
		f.a1 = q + 1 - (q & 1);
	} else {
		f.a0 = f.a1 = q + (fr > 0.5f ? 1 : 0);
	}
	return f;
}

// A block of 256 elements in shared memory (16-byte aligned, zeros behind the row's end), cum the running sum before it. The
// elements are added one by one, by every lane of the warp alike. Returns the first index with fl(cum + p[0] + ... + p[i]) >= randf
// inside the block or -1; cum becomes the sum behind the last element consumed. p >= 0: the sum never decreases, so a group of 32
// is searched only when its last partial sum has reached randf (or is NaN: then maybe none has). The chain of additions is
// what bounds it: 1200 clk with the next 32 elements on their way, 3200 with the next 8. (A scan of the elements' maps per binade
// takes 1900 clk, twice for one change of the binade.)
constexpr int CDF_BLK = 256;
__device__ __forceinline__ int cdf_cross_block(const float *p, float &cum, float randf) {
	const uint32_t s = uint32_t(__cvta_generic_to_shared(p));
	auto load = [&](float4 (&v)[8], int i) {
#pragma unroll
		for (int k = 0; k < 8; k++)
			asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[k].x), "=f"(v[k].y), "=f"(v[k].z), "=f"(v[k].w) : "r"(s + 4u * i + 16u * k) : "memory");
	};
	auto add = [&](const float4 (&v)[8], float c) {
#pragma unroll
		for (int k = 0; k < 8; k++) c = (((c + v[k].x) + v[k].y) + v[k].z) + v[k].w;
		return c;
	};
	float4 a[8], b[8];
	load(a, 0);
	float c = cum;
#pragma unroll 1
	for (int i = 0; i < CDF_BLK; i += 64) {
		float before = c;
		load(b, i + 32);
		c = add(a, c);
		int at = i;
		if (c < randf) {
			before = c;
			if (i + 64 < CDF_BLK) load(a, i + 64);
			c = add(b, c);
			at = i + 32;
		}
		if (!(c < randf)) {  // in the 32 elements from `at` on
#pragma unroll 1
			for (int k = at; k < at + 32; k++) {
				before += p[k];
				if (before >= randf) {
					cum = before;
					return k;
				}
			}
			if (at == i) {  // (a NaN: nothing is reached any more, but the chain goes on)
				if (i + 64 < CDF_BLK) load(a, i + 64);
				c = add(b, c);
			}
		}
	}
	cum = c;
	return -1;
}

// ops::minp_logits, reference ops.hpp:762-859.
//  (1) x /= temp  (2) rowmax  (3) p = exp(x - rowmax), maxp  (4) cut = minp*maxp,
//  denom = sum of p >= cut  (5) every p *= 1/denom — tokens under the cut keep
//  their mass, only the denominator is masked  (6) first index whose running
//  fp32 sum reaches randf, else 0.
// Steps 1-5 are data-parallel. Step 6 must reproduce a *sequential* fp32 sum
// (fp32 addition is not associative, and the crossing index depends on the
// rounding): the maps above evaluate that chain exactly, in parallel
// (cdf_walk_maps, cdf_walk_row).

// Any number of rows, each spread over V / SR_PART CTAs: four kernels (row maximum; exponentials and segment sums;
// scaling and segment maps; the walk). One CTA per row took ~1 ms for a row of 262144: four passes over 1 MB and
// the whole chain of step 6, all latency. Step 6 here: the row is cut into segments of 1024. The sum at a segment's
// start is known approximately from the segment sums, so its binade is, and with it the segment's composite map of that
// binade (see above), which all segments, and all blocks of 256, compute at once. The walk then applies whole segments, 32 at
// a time by a warp scan, and checks every one against the exact state: a segment whose predicted binade is not the actual
// one, or inside which the sum leaves the binade or reaches randf, is walked by its blocks, such a block by its elements.
constexpr int SR_SEG = 1024;
struct MinpRows {
	float *part_max;  // [B][V / SR_PART]
	float2 *seg_sum;  // [B][V / SR_SEG] masked sum, whole sum
	int4 *seg_map;    // [B][V / SR_SEG] a0, a1, exponent of the binade
	int4 *blk_map;    // [B][V / CDF_BLK]
	// step 6 by itself (tg_inverse_cdf): the running sum before the row, and where the sum at its end goes; a sampler has 0 and null
	float cum0;
	float *cum_out;
};
__global__ void __launch_bounds__(SR_THREADS) minp_max_kernel(SampleArgs a, MinpRows w) {
	pdl_trigger();
	pdl_wait();
	__shared__ float red[SR_THREADS / 32];
	const int b = blockIdx.y, tid = threadIdx.x;
	const float *x = a.logits + size_t(b) * a.V + size_t(blockIdx.x) * SR_PART;
	float mx = -INFINITY;
#pragma unroll
	for (int j = 0; j < SR_PART / (4 * SR_THREADS); j++) {
		const float4 v = __ldcg(reinterpret_cast<const float4 *>(x) + tid + SR_THREADS * j);
		mx = fmaxf(mx, fmaxf(fmaxf(v.x / a.temp, v.y / a.temp), fmaxf(v.z / a.temp, v.w / a.temp)));
	}
	mx = warp_max(mx);
	if ((tid & 31) == 0) red[tid >> 5] = mx;
	__syncthreads();
	if (tid == 0) {
		for (int i = 1; i < SR_THREADS / 32; i++) mx = fmaxf(mx, red[i]);
		w.part_max[size_t(b) * gridDim.x + blockIdx.x] = mx;
	}
}
// a warp takes one segment
__global__ void __launch_bounds__(SR_THREADS) minp_exp_kernel(SampleArgs a, MinpRows w) {
	pdl_trigger();
	pdl_wait();
	const int b = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int seg = blockIdx.x * (SR_PART / SR_SEG) + warp;
	float4 *x = reinterpret_cast<float4 *>(a.logits + size_t(b) * a.V + size_t(seg) * SR_SEG);
	float4 v[SR_SEG / 128];
#pragma unroll
	for (int j = 0; j < SR_SEG / 128; j++) v[j] = __ldcg(x + lane + 32 * j);
	float rowmax = -INFINITY;
	for (int c = lane; c < int(gridDim.x); c += 32) rowmax = fmaxf(rowmax, w.part_max[size_t(b) * gridDim.x + c]);
	rowmax = warp_max(rowmax);
	const float cut = a.minp * expf(rowmax - rowmax);  // the largest probability is exp(0)
	float ds = 0.0f, us = 0.0f;
#pragma unroll
	for (int j = 0; j < SR_SEG / 128; j++) {
		v[j].x = expf(v[j].x / a.temp - rowmax);
		v[j].y = expf(v[j].y / a.temp - rowmax);
		v[j].z = expf(v[j].z / a.temp - rowmax);
		v[j].w = expf(v[j].w / a.temp - rowmax);
		__stcg(x + lane + 32 * j, v[j]);
		us += (v[j].x + v[j].y) + (v[j].z + v[j].w);
		ds += (v[j].x < cut) ? 0.0f : v[j].x;
		ds += (v[j].y < cut) ? 0.0f : v[j].y;
		ds += (v[j].z < cut) ? 0.0f : v[j].z;
		ds += (v[j].w < cut) ? 0.0f : v[j].w;
	}
	ds = warp_sum(ds);
	us = warp_sum(us);
	if (lane == 0) w.seg_sum[size_t(b) * (a.V / SR_SEG) + seg] = make_float2(ds, us);
}
// compose the maps of a warp's lanes in lane order; every lane gets the whole
__device__ __forceinline__ CdfFn cdf_warp_compose(CdfFn f) {
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		CdfFn g;
		g.a0 = __shfl_down_sync(0xffffffffu, f.a0, o);
		g.a1 = __shfl_down_sync(0xffffffffu, f.a1, o);
		f = cdf_compose(f, g);  // (right for the lanes whose group of 2 o starts with them: lane 0 in the end)
	}
	f.a0 = __shfl_sync(0xffffffffu, f.a0, 0);
	f.a1 = __shfl_sync(0xffffffffu, f.a1, 0);
	return f;
}
__global__ void __launch_bounds__(SR_THREADS) minp_scale_kernel(SampleArgs a, MinpRows w) {
	pdl_trigger();
	pdl_wait();
	__shared__ float red[SR_THREADS / 32];
	__shared__ float s_pre[SR_THREADS / 32];
	const int b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int nseg = a.V / SR_SEG, seg = blockIdx.x * (SR_PART / SR_SEG) + warp;
	float4 *x = reinterpret_cast<float4 *>(a.logits + size_t(b) * a.V + size_t(seg) * SR_SEG);
	// element order inside the segment: blocks of 256, 8 consecutive ones per lane
	float4 v[2 * (SR_SEG / 256)];
#pragma unroll
	for (int q = 0; q < SR_SEG / 256; q++) {
		v[2 * q] = __ldcg(x + 64 * q + 2 * lane);
		v[2 * q + 1] = __ldcg(x + 64 * q + 2 * lane + 1);
	}
	// the denominator (the same order in every CTA), and what lies before this CTA's first segment
	const float2 *ss = w.seg_sum + size_t(b) * nseg;
	const int first = blockIdx.x * (SR_PART / SR_SEG);
	float ds = 0.0f, us = 0.0f;
	for (int i = tid; i < nseg; i += SR_THREADS) {
		const float2 t = ss[i];
		ds += t.x;
		us += i < first ? t.y : 0.0f;
	}
	ds = warp_sum(ds);
	us = warp_sum(us);
	if (lane == 0) {
		red[warp] = ds;
		s_pre[warp] = us;
	}
	__syncthreads();
	float denom = 0.0f, before = w.cum0;
#pragma unroll
	for (int i = 0; i < SR_THREADS / 32; i++) {
		denom += red[i];
		before += s_pre[i];
	}
	for (int i = first; i < seg; i++) before += ss[i].y;
	const float inv = 1.0f / denom;
	CdfFn whole{0, 0};
	int es = 0;  // the binade of all blocks so far, or -1000
#pragma unroll
	for (int q = 0; q < SR_SEG / CDF_BLK; q++) {
		const float at = before * inv;
		const int e = int((__float_as_uint(at) >> 23) & 0xffu) - 127;
		const bool usable = at >= 7.888609e-31f && e <= 120;
		const float inv_u = usable ? __uint_as_float(unsigned(23 - e + 127) << 23) : 1.0f;
		CdfFn f{0, 0};
		float sum = 0.0f;
#pragma unroll
		for (int h = 0; h < 2; h++) {
			float4 &t = v[2 * q + h];
			sum += (t.x + t.y) + (t.z + t.w);
			t.x *= inv;
			t.y *= inv;
			t.z *= inv;
			t.w *= inv;
			__stcg(x + 64 * q + 2 * lane + h, t);
			f = cdf_compose(f, cdf_element(t.x, inv_u));
			f = cdf_compose(f, cdf_element(t.y, inv_u));
			f = cdf_compose(f, cdf_element(t.z, inv_u));
			f = cdf_compose(f, cdf_element(t.w, inv_u));
		}
		f = cdf_warp_compose(f);
		before += warp_sum(sum);
		whole = cdf_compose(whole, f);
		const int eq = usable ? e : -1000;
		es = q == 0 || es == eq ? eq : -1000;
		if (lane == 0) w.blk_map[(size_t(b) * nseg + seg) * (SR_SEG / CDF_BLK) + q] = make_int4(f.a0, f.a1, eq, 0);
	}
	if (lane == 0) w.seg_map[size_t(b) * nseg + seg] = make_int4(whole.a0, whole.a1, es, 0);
}
// One warp applies the maps get(i) = (a0, a1, binade) of whole segments from `seg` on to the running sum, 32 at a time, up to the first
// one whose binade is not the actual one or inside which the sum leaves the binade or reaches randf.
template <class Get> __device__ __forceinline__ float cdf_walk_maps(Get get, int nseg, float randf, float cum, int &seg) {
	const int lane = threadIdx.x & 31;
	while (seg < nseg) {
		const int4 m = seg + lane < nseg ? get(seg + lane) : make_int4(0, 0, -2000, 0);
		const int e = int((__float_as_uint(cum) >> 23) & 0xffu) - 127;
		if (!(cum >= 7.888609e-31f) || e > 120) break;
		const float u = __uint_as_float(unsigned(e - 23 + 127) << 23), inv_u = __uint_as_float(unsigned(23 - e + 127) << 23);
		const int S0 = int(cum * inv_u);
		const float y = randf * inv_u;
		const int Tmin = min((y < 33554432.0f) ? int(ceilf(y)) : CDF_BIG, 1 << 24);
		CdfFn inc{m.x, m.y};
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			CdfFn prev;
			prev.a0 = __shfl_up_sync(0xffffffffu, inc.a0, o);
			prev.a1 = __shfl_up_sync(0xffffffffu, inc.a1, o);
			if (lane >= o) inc = cdf_compose(prev, inc);
		}
		const int S = cdf_apply(inc, S0);
		const unsigned bad = __ballot_sync(0xffffffffu, m.z != e || S >= Tmin);
		const int n = bad ? __ffs(bad) - 1 : 32;
		if (n > 0) cum = float(__shfl_sync(0xffffffffu, S, n - 1)) * u;
		seg += n;
		if (n < 32) break;
	}
	return cum;
}
// One warp walks a row p of V elements in segments of seg_len (nb blocks of CDF_BLK, the last segment may end early): segment
// maps, inside a segment whose map does not hold the maps of its blocks, inside such a block its elements. cum: the running sum
// before the row, then at the end of the walk. Returns the crossing index, 0 if there is none. chunk: CDF_BLK floats of shared memory.
template <class Seg, class Blk>
__device__ __forceinline__ int cdf_walk_row(Seg seg_map, Blk blk_map, const float *p, int V, int seg_len, int nb, float randf, float &cum, float *chunk) {
	const int lane = threadIdx.x & 31, nseg = (V + seg_len - 1) / seg_len;
#pragma unroll 1
	for (int c = 0; c < nseg; c++) {
		cum = cdf_walk_maps(seg_map, nseg, randf, cum, c);
		if (c >= nseg) break;
		const int m = min(seg_len, V - c * seg_len), mb = (m + CDF_BLK - 1) / CDF_BLK;
#pragma unroll 1
		for (int b = 0; b < mb; b++) {
			cum = cdf_walk_maps([&](int i) { return blk_map(c * nb + i); }, mb, randf, cum, b);
			if (b >= mb) break;
			const int left = min(CDF_BLK, m - CDF_BLK * b);
			__syncwarp();
			{
				const float4 *src = reinterpret_cast<const float4 *>(p + size_t(c) * seg_len + CDF_BLK * b + 8 * lane);
				const float4 z = make_float4(0.f, 0.f, 0.f, 0.f), v0 = 8 * lane < left ? __ldcg(src) : z, v1 = 8 * lane < left ? __ldcg(src + 1) : z;
				reinterpret_cast<float4 *>(chunk + 8 * lane)[0] = v0;
				reinterpret_cast<float4 *>(chunk + 8 * lane)[1] = v1;
			}
			__syncwarp();
			const int r = cdf_cross_block(chunk, cum, randf);
			if (r >= 0) return c * seg_len + CDF_BLK * b + r;
		}
	}
	return 0;
}
// one warp walks a row; the CTA brings the row's maps into shared memory before (minp_walk_smem(V) bytes): the walk is a chain of
// dependent steps, and a load from the L2 in each would double it. Rows whose maps pass 44 KB (staged = 0) are read there.
inline size_t minp_walk_smem(int V) { return size_t(V / SR_SEG) * (1 + SR_SEG / CDF_BLK) * 16; }
__global__ void __launch_bounds__(SR_THREADS) minp_walk_kernel(SampleArgs a, MinpRows w, int staged) {
	pdl_trigger();
	pdl_wait();
	extern __shared__ __align__(16) int4 mw_maps[];  // [nseg] segments, [nseg][NB] blocks
	__shared__ __align__(16) float chunk[CDF_BLK];
	constexpr int NB = SR_SEG / CDF_BLK;
	const int b = blockIdx.x, tid = threadIdx.x;
	const int nseg = a.V / SR_SEG;
	const float *x = a.logits + size_t(b) * a.V;
	auto map = [&](int i) { return __ldcg(i < nseg ? w.seg_map + size_t(b) * nseg + i : w.blk_map + size_t(b) * nseg * NB + (i - nseg)); };
	if (staged) {
#pragma unroll 4
		for (int i = tid; i < nseg * (1 + NB); i += SR_THREADS) mw_maps[i] = map(i);
	}
	float randf = 0.0f;
	const int rc = a.randf_count[b];
	if (rc < a.randf_cap) randf = a.randf[size_t(rc) * a.B + b];
	__syncthreads();
	if (tid >= 32) return;
	float cum = w.cum0;
	const int found = cdf_walk_row([&](int i) { return staged ? mw_maps[i] : map(i); }, [&](int i) { return staged ? mw_maps[nseg + i] : map(nseg + i); }, x, a.V, SR_SEG, NB, randf, cum, chunk);
	if (tid == 0) {
		if (w.cum_out) w.cum_out[b] = cum;
		emit_token(a, b, found);
		a.randf_count[b] = rc + 1;
	}
}

// ------------------------------------------------------------------ min-p of one row by a whole grid
// Steps (3) to (6) for a kernel of G CTAs that can meet at a grid barrier (`sync`): CTA c owns the columns
// [c * cols, (c + 1) * cols), a warp of it blocks of 256. The CTA leaves its masked and whole sum, then (the denominator and
// the approximate sum before every block being known) the composite map of every block in the binade that the running sum
// is expected in, and the map of all its columns where that is one binade. One warp of every CTA then walks the row: CTA
// maps, inside a CTA whose map does not hold the block maps, inside such a block its elements (about 20 blocks of 1024: where the
// sum changes its binade, and the last one). So every CTA knows the token without another exchange. The row was walked
// element by element by one CTA in rounds of 3072 before: a token of the 1B model 829 us for a crossing index in the middle
// of the row, now 740 (695 for the arg-max).
// part: minp_grid_part_bytes(V, G) bytes, of which the first G floats are the caller's; sm: shared memory, minp_grid_floats(V, G)
// floats, 16-byte aligned; red: 2 * NW floats. V is a multiple of 128.
__host__ __device__ __forceinline__ int minp_grid_cols(int V, int G) { return (V / 128 + G - 1) / G * 128; }
__host__ __device__ __forceinline__ int minp_grid_blocks(int V, int G) { return (minp_grid_cols(V, G) + CDF_BLK - 1) / CDF_BLK; }
__host__ __device__ __forceinline__ int minp_grid_floats(int V, int G) {
	const int nb = minp_grid_blocks(V, G);
	return CDF_BLK * nb + 4 * G * (1 + nb) + (nb + 3) / 4 * 4;
}
__host__ __device__ __forceinline__ size_t minp_grid_part_bytes(int V, int G) { return size_t((3 * G + 3) / 4 * 4 + 4 * G * (1 + minp_grid_blocks(V, G))) * 4; }
template <int NW, class Sync>
__device__ __forceinline__ int minp_grid_row(const float *logits, float *probs, int V, float minp, float temp, float gmax, float randf, float *part,
                                             float *sm, float *red, int *scratch, Sync sync) {
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cta = blockIdx.x, G = gridDim.x;
	const int cols = minp_grid_cols(V, G), nb = minp_grid_blocks(V, G), c0 = min(V, cta * cols), n = min(V, c0 + cols) - c0;
	float *pl = sm;                                              // [nb][256]
	int4 *maps = reinterpret_cast<int4 *>(sm + CDF_BLK * nb);    // [G] per CTA, [G][nb] per block
	float *blk = reinterpret_cast<float *>(maps + G * (1 + nb));  // [nb] sums of this CTA's blocks
	int4 *gmaps = reinterpret_cast<int4 *>(part + (3 * G + 3) / 4 * 4);
	// p = exp(z - max); the largest is exp(0), so the cut is minp * exp(gmax - gmax)
	const float cut = minp * expf(gmax - gmax);
	float ds = 0.0f, us = 0.0f;
#pragma unroll 1
	for (int b = warp; b < nb; b += NW) {
		float s = 0.0f;
		if (CDF_BLK * b + 8 * lane < n) {
			float4 v[2];
#pragma unroll
			for (int h = 0; h < 2; h++) v[h] = __ldcg(reinterpret_cast<const float4 *>(logits + c0 + CDF_BLK * b + 8 * lane) + h);
#pragma unroll
			for (int h = 0; h < 2; h++) {
				v[h].x = expf(v[h].x / temp - gmax);
				v[h].y = expf(v[h].y / temp - gmax);
				v[h].z = expf(v[h].z / temp - gmax);
				v[h].w = expf(v[h].w / temp - gmax);
				*(reinterpret_cast<float4 *>(pl + CDF_BLK * b + 8 * lane) + h) = v[h];
				s += (v[h].x + v[h].y) + (v[h].z + v[h].w);
				ds += (v[h].x < cut) ? 0.0f : v[h].x;
				ds += (v[h].y < cut) ? 0.0f : v[h].y;
				ds += (v[h].z < cut) ? 0.0f : v[h].z;
				ds += (v[h].w < cut) ? 0.0f : v[h].w;
			}
		}
		s = warp_sum(s);
		if (lane == 0) blk[b] = s;
		us += s;
	}
	ds = warp_sum(ds);
	__syncthreads();
	if (lane == 0) {
		red[warp] = ds;
		red[NW + warp] = us;
	}
	__syncthreads();
	if (tid == 0) {
		ds = us = 0.0f;
		for (int w = 0; w < NW; w++) {
			ds += red[w];
			us += red[NW + w];
		}
		__stcg(part + G + cta, ds);
		__stcg(part + 2 * G + cta, us);
	}
	sync();
	if (warp == 0) {
		float dv = 0.0f, bv = 0.0f;
		for (int cb = lane; cb < G; cb += 32 * 5) {  // (five loads of each row in flight)
			float d[5], u[5];
#pragma unroll
			for (int q = 0; q < 5; q++) {
				const int c = cb + 32 * q;
				d[q] = c < G ? __ldcg(part + G + c) : 0.0f;
				u[q] = c < cta ? __ldcg(part + 2 * G + c) : 0.0f;
			}
#pragma unroll
			for (int q = 0; q < 5; q++) {
				dv += d[q];
				bv += u[q];
			}
		}
		dv = warp_sum(dv);
		bv = warp_sum(bv);
		if (lane == 0) {
			red[0] = 1.0f / dv;
			red[1] = bv;
		}
	}
	__syncthreads();
	const float inv = red[0];
#pragma unroll 1
	for (int b = warp; b < nb; b += NW) {
		float before = red[1];
		for (int q = 0; q < b; q++) before += blk[q];
		before *= inv;
		const int e = int((__float_as_uint(before) >> 23) & 0xffu) - 127;
		const bool usable = before >= 7.888609e-31f && e <= 120;
		const float inv_u = usable ? __uint_as_float(unsigned(23 - e + 127) << 23) : 1.0f;
		CdfFn f{0, 0};
		if (CDF_BLK * b + 8 * lane < n) {
#pragma unroll
			for (int h = 0; h < 2; h++) {
				float4 t = *(reinterpret_cast<const float4 *>(pl + CDF_BLK * b + 8 * lane) + h);
				t.x *= inv;
				t.y *= inv;
				t.z *= inv;
				t.w *= inv;
				__stcg(reinterpret_cast<float4 *>(probs + c0 + CDF_BLK * b + 8 * lane) + h, t);
				f = cdf_compose(f, cdf_element(t.x, inv_u));
				f = cdf_compose(f, cdf_element(t.y, inv_u));
				f = cdf_compose(f, cdf_element(t.z, inv_u));
				f = cdf_compose(f, cdf_element(t.w, inv_u));
			}
		}
		f = cdf_warp_compose(f);
		if (lane == 0) {
			const int4 m = make_int4(f.a0, f.a1, usable ? e : -1000, 0);
			maps[b] = m;
			__stcg(gmaps + G + cta * nb + b, m);
		}
	}
	__syncthreads();
	if (tid == 0) {
		CdfFn whole{0, 0};
		int e = maps[0].z;
		for (int b = 0; CDF_BLK * b < n; b++) {
			whole = cdf_compose(whole, CdfFn{maps[b].x, maps[b].y});
			if (maps[b].z != e) e = -1000;
		}
		__stcg(gmaps + cta, make_int4(whole.a0, whole.a1, e, 0));
	}
	sync();
	for (int c = tid; c < G * (1 + nb); c += 32 * NW) maps[c] = __ldcg(gmaps + c);
	__syncthreads();
	if (warp == 0) {
		float cum = 0.0f;
		const int found = cdf_walk_row([&](int i) { return maps[i]; }, [&](int i) { return maps[G + i]; }, probs, V, cols, nb, randf, cum, pl);
		if (lane == 0) scratch[0] = found;
	}
	__syncthreads();
	const int found = scratch[0];
	__syncthreads();
	return found;
}

// ------------------------------------------------------------------ grid-wide min-p (one sequence)
// ops::minp_logits for a single row spread over G CTAs of SG_THREADS threads (cooperative launch: the
// CTAs meet at a bounded grid barrier). It partitions the row and orders every floating-point sum exactly like the
// sampler inside the persistent decode kernels (minp_grid_row), so a token sampled step by step (tg_decode +
// tg_sample_minp) is the token the device-resident loop samples. The row is overwritten with the probabilities, as the
// reference does.
constexpr int SG_THREADS = 384;
constexpr int SG_NWARPS = SG_THREADS / 32;
constexpr int SG_SPIN_CAP = 1 << 22;

__device__ __forceinline__ bool sg_grid_sync(unsigned *bar, unsigned &epoch, unsigned G, int *fail) {
	__syncthreads();
	epoch += 1;
	if (threadIdx.x == 0 && !*(volatile int *)fail) {
		__threadfence();
		const unsigned old = atomicAdd(bar, 1u);
		if (old + 1u < epoch * G) {
			int spins = 0;
			unsigned v;
			do {
				asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
			} while (v < epoch * G && ++spins < SG_SPIN_CAP);
			if (v < epoch * G) *fail = 1;  // the wait ran out: everybody falls through from here on
		}
	}
	__syncthreads();
	return !*(volatile int *)fail;
}

// part: minp_grid_part_bytes(V, G) of scratch, bar: one zeroed word, err: error word, minp_grid_floats(V, G) dynamic floats
__global__ void __launch_bounds__(SG_THREADS, 1) minp_grid_kernel(SampleArgs a, unsigned *bar, float *part, int *err) {
	extern __shared__ __align__(16) float sm[];
	__shared__ float red[2 * SG_NWARPS];
	__shared__ int scratch[1];
	__shared__ float s_max;
	__shared__ int s_fail;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int cta = blockIdx.x, G = gridDim.x;
	const int cols = minp_grid_cols(a.V, G), c0 = min(a.V, cta * cols), c1 = min(a.V, c0 + cols);
	unsigned epoch = 0;
	if (tid == 0) s_fail = 0;
	__syncthreads();
	// (1)+(2) row maximum of z = logit / temp
	float mx = -INFINITY;
#pragma unroll 2
	for (int i = c0 + 4 * tid; i < c1; i += 4 * SG_THREADS) {
		const float4 v = __ldcg(reinterpret_cast<const float4 *>(a.logits + i));
		mx = fmaxf(mx, fmaxf(fmaxf(v.x / a.temp, v.y / a.temp), fmaxf(v.z / a.temp, v.w / a.temp)));
	}
	mx = warp_max(mx);
	if (lane == 0) red[warp] = mx;
	__syncthreads();
	if (tid == 0) {
		float m = red[0];
		for (int w = 1; w < SG_NWARPS; w++) m = fmaxf(m, red[w]);
		__stcg(part + cta, m);
	}
	sg_grid_sync(bar, epoch, G, &s_fail);
	if (warp == 0) {
		float m = -INFINITY;
#pragma unroll 1
		for (int c = lane; c < G; c += 32) m = fmaxf(m, __ldcg(part + c));
		m = warp_max(m);
		if (lane == 0) s_max = m;
	}
	__syncthreads();
	const float gmax = s_max;
	const int rc = a.randf_count[0];  // (read by every CTA before the barriers behind which CTA 0 counts up)
	const float randf = rc < a.randf_cap ? a.randf[size_t(rc) * a.B] : 0.0f;
	// (3) to (6); every probability is scaled in place of its logit
	const int tok = minp_grid_row<SG_NWARPS>(a.logits, a.logits, a.V, a.minp, a.temp, gmax, randf, part, sm, red, scratch,
	                                         [&] { sg_grid_sync(bar, epoch, G, &s_fail); });
	if (cta == 0 && tid == 0 && !*(volatile int *)&s_fail) {
		emit_token(a, 0, tok);
		a.randf_count[0] = rc + 1;
	}
	if (tid == 0 && *(volatile int *)&s_fail) atomicExch(err, 8);
}

}  // namespace tg
