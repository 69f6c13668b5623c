// Attention over fp32 K / V rows on the CUDA cores, for the shapes whose time is latency and memory traffic, not
// arithmetic: one decode step per sequence, and short prompts.
//
// The rows of a sequence's keys (values) follow each other in memory, so a chunk of 32 keys is ONE bulk copy of 32 KB
// into shared memory: the whole traffic of a CTA is asynchronous and costs no registers. A buffer is filled again as soon
// as its scores (K) or products (V) are done.
// The prefill kernel's step over a chunk: scores (a warp takes a few keys against all query rows; a lane holds 8 of the 256 dimensions, and the
// lanes' partial sums meet in a reduce-scatter, one shuffle per score), one softmax step per query row with lane = key,
// then the products with V (a thread holds 4 dimensions of every row for a share of the keys).
//
// The result leaves as the digits of the O projection's operand (kernels_gemm_i8.cuh) where the caller wants them: the
// CTA that finishes a row has all of it.
#pragma once
#include "kernels_decode.cuh"  // AT_NH, AT_HD
#include "kernels_gemm_i8.cuh"
#include "tg_common.cuh"

namespace tg {

constexpr int AC_KEYS = 32;
constexpr int AC_BUF = AC_KEYS * 1024;  // bytes of a K or V chunk
constexpr int AC_SMEM = 2 * AC_BUF;

// N partial sums per lane (N = 16): afterwards lane L holds the warp's total of value L >> 1
__device__ __forceinline__ float ac_reduce16(float (&t)[16], int lane) {
#pragma unroll
	for (int o = 8; o >= 1; o >>= 1) {
		const bool up = lane & (2 * o);
#pragma unroll
		for (int i = 0; i < o; i++) {
			const float keep = up ? t[i + o] : t[i], send = up ? t[i] : t[i + o];
			t[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * o);
		}
	}
	return t[0] + __shfl_xor_sync(0xffffffffu, t[0], 1);
}
__device__ __forceinline__ float ac_dot8(const float4 &q0, const float4 &q1, const float4 &k0, const float4 &k1) {
	float t = q0.x * k0.x;
	t = fmaf(q0.y, k0.y, t);
	t = fmaf(q0.z, k0.z, t);
	t = fmaf(q0.w, k0.w, t);
	t = fmaf(q1.x, k1.x, t);
	t = fmaf(q1.y, k1.y, t);
	t = fmaf(q1.z, k1.z, t);
	return fmaf(q1.w, k1.w, t);
}
// the same two products per instruction (the two halves are added at the end)
__device__ __forceinline__ float ac_dot8x2(const float4 &q0, const float4 &q1, const float4 &k0, const float4 &k1) {
	float2 t = make_float2(q0.x * k0.x, q0.y * k0.y);
	t = ffma2(make_float2(q0.z, q0.w), make_float2(k0.z, k0.w), t);
	t = ffma2(make_float2(q1.x, q1.y), make_float2(k1.x, k1.y), t);
	t = ffma2(make_float2(q1.z, q1.w), make_float2(k1.z, k1.w), t);
	return t.x + t.y;
}
__device__ __forceinline__ void ac_fma4x2(float4 &o, float p, const float4 &v) {
	const float2 pp = make_float2(p, p), lo = ffma2(pp, make_float2(v.x, v.y), make_float2(o.x, o.y)), hi = ffma2(pp, make_float2(v.z, v.w), make_float2(o.z, o.w));
	o = make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ void ac_fma4(float4 &o, float p, const float4 &v) {
	o.x = fmaf(p, v.x, o.x);
	o.y = fmaf(p, v.y, o.y);
	o.z = fmaf(p, v.z, o.z);
	o.w = fmaf(p, v.w, o.w);
}

// ------------------------------------------------------------------ decode: one query per sequence
struct AttnArgs {
	const float *qkv;   // [B][1536] = q(4x256) | k(256) | v(256)
	// qkv_nsplit > 0: qkv instead holds the raw K-split partial sums of the grouped q|k|v GEMM,
	// [qkv_nsplit][B][1536], and sq / sk / sv are the column scales (splits are added in ascending order)
	int qkv_nsplit, qkv_B;
	const float *sq, *sk, *sv;
	const float *rmsq;  // [256]
	const float *rmsk;  // [256]
	const float *cosT;  // [n_pos][256]
	const float *sinT;
	float *kcache;      // [B][slots][256]
	float *vcache;
	int slots;          // 512 on local layers, max_pos_global on global layers
	int is_local;
	const int *step_pos;   // [B]
	const int *ring_base;  // [B] prompt length if it filled the ring, else 0 (decode.hpp:98-103)
	float *part;        // [B][nsplit][4*256 + 8]
	unsigned *tickets;  // [B]
	float *out;         // [B][1024], or null:
	uint8_t *x;         // the digits of the result (K = 1024) and their row scales
	float *rowscale;
	int groups;
	int nsplit;
	int *err_flag;
};
constexpr int AT_THREADS = 256;
constexpr int AT_PART = AT_NH * AT_HD + 8;
// A step reads every cached row once: HBM bounds it for many sequences, the chain of dependent round trips for few.
// A warp takes 4 keys of every 32 against all four heads and runs on its own through a ring of three 4 KB buffers (K, V,
// K, V, ..), with its own running maximum: nothing in the loop waits for another warp. The ring keeps 64 to 96 KB per CTA
// in flight, two CTAs per SM (HBM's rate times its latency under load is ~70 KB per SM). 256 sequences of 182 keys, 94 MB:
// 33.5 us with one K and one V buffer and block-wide steps over 32 keys and two splits, 23 us now.
constexpr int AD_KEYS = 4, AD_ROUND = AD_KEYS * AT_THREADS / 32;
constexpr int AD_BUF = AD_KEYS * 1024;
constexpr int AD_STAGES = 3;
constexpr int AD_SMEM = AT_THREADS / 32 * AD_STAGES * AD_BUF;

__global__ void __launch_bounds__(AT_THREADS, 2) attn_decode_kernel(AttnArgs a) {
	extern __shared__ __align__(128) uint8_t ac_smem[];
	__shared__ __align__(16) float rowbuf[AT_NH * AT_HD + 2 * AT_HD];  // q | k | v of the new token, normed and rotated
	__shared__ float m_s[AT_THREADS / 32][AT_NH], l_s[AT_THREADS / 32][AT_NH];
	__shared__ uint64_t full[AT_THREADS / 32][AD_STAGES];
	__shared__ uint32_t red[AT_THREADS / 32];
	__shared__ int s_last;
	const int b = blockIdx.y, split = blockIdx.x;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	uint8_t *ring = ac_smem + warp * (AD_STAGES * AD_BUF);
	if (lane == 0) {
		for (int i = 0; i < AD_STAGES; i++) mbar_init(&full[warp][i], 1);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	__syncwarp();
	// the weights are nobody's output: requested before the wait for the predecessor. Warps 0..3: a head of q, 4: k, 5: v
	constexpr int NQ = AT_NH * AT_HD + 2 * AT_HD;
	const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
	float4 w0 = z4, w1 = z4, s0 = z4, s1 = z4;
	if (warp <= AT_NH) {
		const float4 *w = reinterpret_cast<const float4 *>(warp < AT_NH ? a.rmsq : a.rmsk);
		w0 = __ldg(w + lane);
		w1 = __ldg(w + 32 + lane);
	}
	if (warp < AT_NH + 2 && a.qkv_nsplit > 0) {
		const float4 *scl = reinterpret_cast<const float4 *>(warp < AT_NH ? a.sq + warp * AT_HD : (warp == AT_NH ? a.sk : a.sv));
		s0 = __ldg(scl + lane);
		s1 = __ldg(scl + 32 + lane);
	}
	pdl_trigger();
	pdl_wait();
	int pos = a.step_pos[b];
	const int base = a.is_local ? a.ring_base[b] : 0;
	float4 lo = z4, hi = z4;
	if (warp < AT_NH + 2) {  // (in flight together with the position)
		const float4 *p = reinterpret_cast<const float4 *>(a.qkv + size_t(b) * NQ + warp * AT_HD);
		if (a.qkv_nsplit > 0) {
			const size_t sstride = size_t(a.qkv_B) * (NQ / 4);
			for (int sp = 0; sp < a.qkv_nsplit; sp += 4) {
				float4 u[4], v[4];
#pragma unroll
				for (int q = 0; q < 4; q++) {
					u[q] = v[q] = z4;
					if (sp + q < a.qkv_nsplit) {
						u[q] = p[size_t(sp + q) * sstride + lane];
						v[q] = p[size_t(sp + q) * sstride + 32 + lane];
					}
				}
#pragma unroll
				for (int q = 0; q < 4; q++) {
					lo.x += u[q].x;
					lo.y += u[q].y;
					lo.z += u[q].z;
					lo.w += u[q].w;
					hi.x += v[q].x;
					hi.y += v[q].y;
					hi.z += v[q].z;
					hi.w += v[q].w;
				}
			}
			lo = make_float4(lo.x * s0.x, lo.y * s0.y, lo.z * s0.z, lo.w * s0.w);
			hi = make_float4(hi.x * s1.x, hi.y * s1.y, hi.z * s1.z, hi.w * s1.w);
		} else {
			lo = p[lane];
			hi = p[32 + lane];
		}
	}
	int slot, valid;
	if (a.is_local) {
		slot = (pos - base) % a.slots;
		valid = min(pos + 1, a.slots);
	} else {
		if (pos >= a.slots) {  // cache full: refuse to write out of bounds
			if (tid == 0) *a.err_flag = 2;
			pos = a.slots - 1;
		}
		slot = pos;
		valid = pos + 1;
	}
	// whole rounds of 32 keys are dealt out to the splits; splits without any leave at once
	const int rounds = (valid + AD_ROUND - 1) / AD_ROUND, per = (rounds + a.nsplit - 1) / a.nsplit, nact = (rounds + per - 1) / per;
	if (split >= nact) return;
	const int j0 = split * per * AD_ROUND, j1 = min(valid, j0 + per * AD_ROUND);
	const int jw = j0 + AD_KEYS * warp, nit = max(0, (j1 - jw + AD_ROUND - 1) / AD_ROUND);  // this warp's first key, its groups of keys
	float *kc = a.kcache + size_t(b) * a.slots * AT_HD, *vc = a.vcache + size_t(b) * a.slots * AT_HD;
	// item i of the warp's ring: the keys (i even) or the values (i odd) of group i / 2; called by the whole warp
	auto issue = [&](int i) {
		const int j = jw + (i >> 1) * AD_ROUND, st = i % AD_STAGES;
		const uint32_t bytes = uint32_t(min(AD_KEYS, j1 - j)) * 1024u;
		if (i < 2 * nit && tc_elect()) {
			mbar_expect_tx(&full[warp][st], bytes);
			bulk_load(ring + st * AD_BUF, (i & 1 ? vc : kc) + size_t(j) * AT_HD, bytes, &full[warp][st]);
		}
	};
#pragma unroll
	for (int i = 0; i < AD_STAGES; i++) issue(i);
	if (warp <= AT_NH) {  // per-head norm and RoPE; lane owns d = 4 lane .. and the partners 128 + d
		// the reference scales q by 1/sqrt(256) = 2^-4 before the dot products (ops.hpp:262,283)
		const float qs = warp < AT_NH ? 0.0625f : 1.0f;
		const float4 *cr = reinterpret_cast<const float4 *>(a.cosT + size_t(pos) * AT_HD), *sr = reinterpret_cast<const float4 *>(a.sinT + size_t(pos) * AT_HD);
		const float4 c0 = cr[lane], c1 = cr[32 + lane], n0 = sr[lane], n1 = sr[32 + lane];
		const float lov[4] = {lo.x, lo.y, lo.z, lo.w}, hiv[4] = {hi.x, hi.y, hi.z, hi.w};
		const float wlo[4] = {w0.x, w0.y, w0.z, w0.w}, whi[4] = {w1.x, w1.y, w1.z, w1.w};
		const float clo[4] = {c0.x, c0.y, c0.z, c0.w}, chi[4] = {c1.x, c1.y, c1.z, c1.w};
		const float slo[4] = {n0.x, n0.y, n0.z, n0.w}, shi[4] = {n1.x, n1.y, n1.z, n1.w};
		float ss = 0.0f;
#pragma unroll
		for (int i = 0; i < 4; i++) {
			ss = fmaf(lov[i], lov[i], ss);
			ss = fmaf(hiv[i], hiv[i], ss);
		}
		ss = warp_sum(ss);
		const float r = inv_rms(ss, AT_HD);
		float yl[4], yh[4];
#pragma unroll
		for (int i = 0; i < 4; i++) {
			const float u = (lov[i] * r) * (wlo[i] + 1.0f), v = (hiv[i] * r) * (whi[i] + 1.0f);
			// y = cos*x + rotate_half(x)*sin, rotate_half = [-x_hi, x_lo]
			yl[i] = fmaf(-1.0f * v, slo[i], clo[i] * u) * qs;
			yh[i] = fmaf(u, shi[i], chi[i] * v) * qs;
		}
		lo = make_float4(yl[0], yl[1], yl[2], yl[3]);
		hi = make_float4(yh[0], yh[1], yh[2], yh[3]);
	}
	if (warp < AT_NH + 2) {
		float4 *x = reinterpret_cast<float4 *>(&rowbuf[warp * AT_HD]);
		x[lane] = lo;
		x[32 + lane] = hi;
		if (warp >= AT_NH && slot >= j0 && slot < j1) {
			float4 *c = reinterpret_cast<float4 *>((warp == AT_NH ? kc : vc) + size_t(slot) * AT_HD);
			c[lane] = lo;
			c[32 + lane] = hi;
		}
	}
	__syncthreads();
	float4 q0[AT_NH], q1[AT_NH];
#pragma unroll
	for (int h = 0; h < AT_NH; h++) {
		q0[h] = *reinterpret_cast<const float4 *>(&rowbuf[h * AT_HD + 4 * lane]);
		q1[h] = *reinterpret_cast<const float4 *>(&rowbuf[h * AT_HD + 128 + 4 * lane]);
	}
	float4 o0[AT_NH], o1[AT_NH];  // lane: dimensions 4 lane .. and 128 + 4 lane ..
#pragma unroll
	for (int h = 0; h < AT_NH; h++) o0[h] = o1[h] = z4;
	float m = -INFINITY, l = 0.0f;  // of head (lane >> 1) & 3
	// the cache does not hold the new token's row yet (n: 4 for the key row of rowbuf, 5 for the value row)
	auto patch = [&](uint8_t *buf, int at, int n) {
		if (at < 0 || at >= AD_KEYS) return;
		float4 *d = reinterpret_cast<float4 *>(buf + at * 1024);
		const float4 *x = reinterpret_cast<const float4 *>(&rowbuf[n * AT_HD]);
		d[lane] = x[lane];
		d[32 + lane] = x[32 + lane];
		fence_proxy_async();  // (the buffer's next content arrives by a bulk copy)
		__syncwarp();
	};
	int cap = TC_SPIN_CAP;
	for (int it = 0; it < nit; it++) {
		const int j = jw + it * AD_ROUND, n = min(AD_KEYS, j1 - j);
		const int ik = 2 * it, iv = 2 * it + 1;
		uint8_t *K = ring + ik % AD_STAGES * AD_BUF, *V = ring + iv % AD_STAGES * AD_BUF;
		tc_wait_cap(&full[warp][ik % AD_STAGES], ik / AD_STAGES & 1, cap);
		patch(K, slot - j, AT_NH);
		float t[16];
#pragma unroll
		for (int kk = 0; kk < AD_KEYS; kk++) {  // (rows past n hold an older group's keys, or nothing yet: their scores are not used)
			const float4 k0 = *reinterpret_cast<const float4 *>(K + kk * 1024 + 16 * lane), k1 = *reinterpret_cast<const float4 *>(K + kk * 1024 + 512 + 16 * lane);
#pragma unroll
			for (int h = 0; h < AT_NH; h++) t[kk * 4 + h] = ac_dot8(q0[h], q1[h], k0, k1);
		}
		float z = ac_reduce16(t, lane);  // key lane >> 3, head (lane >> 1) & 3
		__syncwarp();
		issue(ik + AD_STAGES);
		if ((lane >> 3) >= n) z = -INFINITY;
		float mn = fmaxf(m, z);
		mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 8));
		mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 16));  // finite: a group has at least one key
		const float p = expf(z - mn), cr = expf(m - mn);
		float ps = p + __shfl_xor_sync(0xffffffffu, p, 8);
		ps += __shfl_xor_sync(0xffffffffu, ps, 16);
		l = fmaf(l, cr, ps);
		m = mn;
		if (__any_sync(0xffffffffu, cr != 1.0f)) {
#pragma unroll
			for (int h = 0; h < AT_NH; h++) {
				const float c = __shfl_sync(0xffffffffu, cr, 2 * h);
				o0[h] = make_float4(o0[h].x * c, o0[h].y * c, o0[h].z * c, o0[h].w * c);
				o1[h] = make_float4(o1[h].x * c, o1[h].y * c, o1[h].z * c, o1[h].w * c);
			}
		}
		tc_wait_cap(&full[warp][iv % AD_STAGES], iv / AD_STAGES & 1, cap);
		patch(V, slot - j, AT_NH + 1);
#pragma unroll
		for (int kk = 0; kk < AD_KEYS; kk++) {
			if (kk < n) {
				const float4 v0 = *reinterpret_cast<const float4 *>(V + kk * 1024 + 16 * lane), v1 = *reinterpret_cast<const float4 *>(V + kk * 1024 + 512 + 16 * lane);
#pragma unroll
				for (int h = 0; h < AT_NH; h++) {
					const float w = __shfl_sync(0xffffffffu, p, 8 * kk + 2 * h);
					ac_fma4(o0[h], w, v0);
					ac_fma4(o1[h], w, v1);
				}
			}
		}
		__syncwarp();
		issue(iv + AD_STAGES);
	}
	if (cap == 0) *static_cast<volatile int *>(a.err_flag) = 6;
	// ---- join the warps: thread (h, d4) ends up with four consecutive outputs
	__syncthreads();  // (every warp has consumed its ring)
	float4 *jb = reinterpret_cast<float4 *>(ac_smem);
#pragma unroll
	for (int h = 0; h < AT_NH; h++) {
		jb[(warp * AT_NH + h) * 64 + lane] = o0[h];
		jb[(warp * AT_NH + h) * 64 + 32 + lane] = o1[h];
	}
	if (lane < 2 * AT_NH && !(lane & 1)) {
		m_s[warp][lane >> 1] = m;
		l_s[warp][lane >> 1] = l;
	}
	__syncthreads();
	const int h = tid >> 6, d4 = tid & 63;
	float Ms = -INFINITY, L = 0.0f;
#pragma unroll
	for (int g = 0; g < AT_THREADS / 32; g++) Ms = fmaxf(Ms, m_s[g][h]);  // finite: warp 0 has a key
	float4 r = z4;
#pragma unroll
	for (int g = 0; g < AT_THREADS / 32; g++) {
		const float w = expf(m_s[g][h] - Ms);
		L = fmaf(l_s[g][h], w, L);
		ac_fma4(r, w, jb[(g * AT_NH + h) * 64 + d4]);
	}
	if (nact > 1) {
		float *pb = a.part + size_t(b) * a.nsplit * AT_PART;
		float *prow = pb + size_t(split) * AT_PART;
		__stcg(reinterpret_cast<float4 *>(prow) + tid, r);
		if (d4 == 0) {
			__stcg(prow + AT_NH * AT_HD + h, Ms);
			__stcg(prow + AT_NH * AT_HD + 4 + h, L);
		}
		__threadfence();
		__syncthreads();
		if (tid == 0) s_last = atomicAdd(&a.tickets[b], 1u) == unsigned(nact - 1);
		__syncthreads();
		if (!s_last) return;
		__threadfence();
		float M = -INFINITY;
		for (int sp = 0; sp < nact; sp++) M = fmaxf(M, __ldcg(pb + size_t(sp) * AT_PART + AT_NH * AT_HD + h));
		r = make_float4(0.f, 0.f, 0.f, 0.f);
		L = 0.0f;
		for (int s0 = 0; s0 < nact; s0 += 4) {
			float4 v[4];
			float ms[4], ls[4];
#pragma unroll
			for (int q = 0; q < 4; q++) {
				v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
				ms[q] = -INFINITY;
				ls[q] = 0.0f;
				if (s0 + q < nact) {
					const float *p = pb + size_t(s0 + q) * AT_PART;
					v[q] = __ldcg(reinterpret_cast<const float4 *>(p) + tid);
					ms[q] = __ldcg(p + AT_NH * AT_HD + h);
					ls[q] = __ldcg(p + AT_NH * AT_HD + 4 + h);
				}
			}
#pragma unroll
			for (int q = 0; q < 4; q++) {
				const float w = expf(ms[q] - M);
				L = fmaf(ls[q], w, L);
				ac_fma4(r, w, v[q]);
			}
		}
		if (tid == 0) a.tickets[b] = 0u;
	}
	r.x /= L;
	r.y /= L;
	r.z /= L;
	r.w /= L;
	if (a.out) {
		reinterpret_cast<float4 *>(a.out + size_t(b) * (AT_NH * AT_HD))[tid] = r;
	} else {
		const uint32_t mb = block_umax<AT_THREADS / 32>(max(max(i8_abs_bits(r.x), i8_abs_bits(r.y)), max(i8_abs_bits(r.z), i8_abs_bits(r.w))), red);
		if (tid == 0) a.rowscale[b] = i8_row_scale(mb);
		i8_pack4(a.x, a.groups, b, tid, r, i8_row_mul(mb));
	}
}

// ------------------------------------------------------------------ prefill of short prompts
// Two queries (8 rows of 4 heads) per CTA of 16 warps; the FMAs and the score reductions bound it (~920 issue slots per 32
// keys and step), so products are packed two to an instruction. q [S][1024], k and v [off + S][256] per prompt; blockIdx.y is the
// prompt. Query s is the token at key off + s (off > 0: a continuation, its context comes first). Causal; on local layers
// a query sees at most `window` keys before itself (the reference's prefill rule, ops.hpp:439-443).
// A cluster of ks CTAs shares two queries, each with a part of their keys (a chunk of 32 keys is a chain of three barriers, ~2 us): the
// first one joins the parts, in key order. attn_small_split: how many.
constexpr int APS_THREADS = 512;
// CTAs per two queries of a prompt of S tokens behind `off` others. By the prompt alone: a prompt of a group gets the bits that it
// gets by itself. Two chunks of keys per CTA at least, and not many more CTAs than are resident (one per SM): 178 tokens 2,
// 61 behind 1500 cached ones 6. (prefill of 178 tokens 1862 -> 1804 us)
inline int attn_small_split(int S, int off, int is_local, int window) {
	const int keys = is_local ? std::min(off + S, window + 2) : off + S;
	return std::max(1, std::min(std::min(8, (keys + AC_KEYS - 1) / AC_KEYS / 2), 192 / ((S + 1) / 2)));
}
__device__ __forceinline__ uint32_t ac_mapa(const void *p, int rank) {
	uint32_t r;
	asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
	return r;
}
__device__ __forceinline__ float ac_remote(const float *p, int rank) {
	float v;
	asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(ac_mapa(p, rank)) : "memory");
	return v;
}
__device__ __forceinline__ float4 ac_remote4(const float4 *p, int rank) {
	float4 v;
	asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(ac_mapa(p, rank)) : "memory");
	return v;
}
__global__ void __launch_bounds__(APS_THREADS, 1) attn_prefill_small_kernel(float *o_out, uint8_t *x, float *rowscale, int groups, const float *q,
                                                                            const float *k, const float *v, int S, int off, int is_local, int window,
                                                                            int ks, int *err) {
	extern __shared__ __align__(128) uint8_t ac_smem[];
	constexpr int R = 8;  // query rows
	__shared__ __align__(16) float sc[AC_KEYS][R], pr[AC_KEYS][R];
	__shared__ float corr_s[R], l_s[R], m_s[R];
	__shared__ uint64_t kbar, vbar;
	__shared__ uint32_t red[APS_THREADS / 32];
	float *K = reinterpret_cast<float *>(ac_smem), *V = reinterpret_cast<float *>(ac_smem + AC_BUF);
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	if (tid == 0) {
		mbar_init(&kbar, 1);
		mbar_init(&vbar, 1);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	__syncthreads();
	pdl_trigger();
	pdl_wait();
	const size_t r0 = size_t(blockIdx.y) * S;
	const int rank = ks > 1 ? int(blockIdx.x) % ks : 0;  // of the cluster's CTAs
	const int s0 = (int(gridDim.x) / ks - 1 - int(blockIdx.x) / ks) * 2;  // (the longest walks start first)
	const int s_last = min(S - 1, s0 + 1);
	const int j0 = (is_local && off + s0 >= window) ? off + s0 - window : 0, j1 = off + s_last + 1;
	// this CTA's chunks: c_lo .. c_lo + nch - 1 of all
	const int all = (j1 - j0 + AC_KEYS - 1) / AC_KEYS, c_lo = all * rank / ks, nch = all * (rank + 1) / ks - c_lo;
	k += (r0 + j0) * 256;  // (a continuation is one sequence: r0 = 0)
	v += (r0 + j0) * 256;
	auto issue = [&](float *dst, const float *src, int c, uint64_t *bar) {
		c += c_lo;
		const uint32_t bytes = uint32_t(min(AC_KEYS, j1 - j0 - c * AC_KEYS)) * 1024u;
		fence_proxy_async();
		mbar_expect_tx(bar, bytes);
		bulk_load(dst, src + size_t(c) * AC_KEYS * 256, bytes, bar);
	};
	if (tid == 0 && nch > 0) {
		issue(K, k, 0, &kbar);
		issue(V, v, 0, &vbar);
	}
	// row = query * 4 + head
	float4 q0[R], q1[R];
#pragma unroll
	for (int r = 0; r < R; r++) {
		const int s = s0 + (r >> 2);
		q0[r] = q1[r] = make_float4(0.f, 0.f, 0.f, 0.f);
		if (s < S) {
			const float4 *qr = reinterpret_cast<const float4 *>(q + (r0 + s) * 1024 + (r & 3) * 256);
			q0[r] = qr[lane];
			q1[r] = qr[32 + lane];
		}
		// exact: the reference scales q by 1/sqrt(256) = 2^-4 before the dot products
		q0[r].x *= 0.0625f; q0[r].y *= 0.0625f; q0[r].z *= 0.0625f; q0[r].w *= 0.0625f;
		q1[r].x *= 0.0625f; q1[r].y *= 0.0625f; q1[r].z *= 0.0625f; q1[r].w *= 0.0625f;
	}
	const int d4 = tid & 63, kg = tid >> 6;  // 8 groups of 4 keys
	float4 o[R];
#pragma unroll
	for (int r = 0; r < R; r++) o[r] = make_float4(0.f, 0.f, 0.f, 0.f);
	float m = -INFINITY, l = 0.0f;  // of row `warp` (warps 0..7)
	for (int c = 0; c < nch; c++) {
		const int base = j0 + (c_lo + c) * AC_KEYS, n = min(AC_KEYS, j1 - base);
		tc_wait(&kbar, c & 1, err);
		{
			float t[16];
#pragma unroll
			for (int kk = 0; kk < 2; kk++) {
				const float4 k0 = *reinterpret_cast<const float4 *>(K + (2 * warp + kk) * 256 + 4 * lane);
				const float4 k1 = *reinterpret_cast<const float4 *>(K + (2 * warp + kk) * 256 + 128 + 4 * lane);
#pragma unroll
				for (int r = 0; r < R; r++) t[kk * 8 + r] = ac_dot8x2(q0[r], q1[r], k0, k1);
			}
			const float z = ac_reduce16(t, lane);
			if (!(lane & 1)) sc[2 * warp + (lane >> 4)][(lane >> 1) & 7] = z;
		}
		__syncthreads();  // scores complete, K consumed
		if (tid == 0 && c + 1 < nch) issue(K, k, c + 1, &kbar);
		if (warp < R) {
			const int s = off + s0 + (warp >> 2), j = base + lane;
			const bool vis = lane < n && j <= s && !(is_local && j + window < s);
			const float z = vis ? sc[lane][warp] : -INFINITY;
			const float mn = fmaxf(m, warp_max(z));
			// (a row may have no visible key in its first chunk: the second query's window starts one later)
			const float p = vis ? expf(z - mn) : 0.0f, cr = m == -INFINITY ? 0.0f : expf(m - mn);
			l = fmaf(l, cr, warp_sum(p));
			m = mn;
			pr[lane][warp] = p;
			if (lane == 0) corr_s[warp] = cr;
		}
		tc_wait(&vbar, c & 1, err);
		__syncthreads();  // probabilities complete
#pragma unroll
		for (int r = 0; r < R; r++) {
			const float cr = corr_s[r];
			o[r].x *= cr;
			o[r].y *= cr;
			o[r].z *= cr;
			o[r].w *= cr;
		}
#pragma unroll
		for (int kk = 0; kk < AC_KEYS / 8; kk++) {
			const int key = kg * (AC_KEYS / 8) + kk;
			if (key < n) {
				const float4 vv = *reinterpret_cast<const float4 *>(V + key * 256 + 4 * d4);
				const float4 pa = *reinterpret_cast<const float4 *>(&pr[key][0]), pb = *reinterpret_cast<const float4 *>(&pr[key][4]);
				ac_fma4x2(o[0], pa.x, vv);
				ac_fma4x2(o[1], pa.y, vv);
				ac_fma4x2(o[2], pa.z, vv);
				ac_fma4x2(o[3], pa.w, vv);
				ac_fma4x2(o[4], pb.x, vv);
				ac_fma4x2(o[5], pb.y, vv);
				ac_fma4x2(o[6], pb.z, vv);
				ac_fma4x2(o[7], pb.w, vv);
			}
		}
		__syncthreads();  // V consumed
		if (tid == 0 && c + 1 < nch) issue(V, v, c + 1, &vbar);
	}
	// ---- join the eight key groups (64 KB: both buffers); thread (query, k4) ends up with 4 of its query's 1024 outputs
	float4 *jb = reinterpret_cast<float4 *>(ac_smem);
#pragma unroll
	for (int r = 0; r < R; r++) jb[(kg * R + r) * 64 + d4] = o[r];
	if (warp < R && lane == 0) {
		l_s[warp] = l;
		m_s[warp] = m;
	}
	__syncthreads();
	const int qi = tid >> 8, k4 = tid & 255, row = qi * 4 + (k4 >> 6);
	float4 r = jb[row * 64 + (k4 & 63)];
#pragma unroll
	for (int g = 1; g < 8; g++) {
		const float4 t = jb[(g * R + row) * 64 + (k4 & 63)];
		r.x += t.x;
		r.y += t.y;
		r.z += t.z;
		r.w += t.w;
	}
	float L = l_s[row];
	if (ks > 1) {  // the other CTAs' parts, through the cluster's shared memory, in key order
		float4 *mine = jb;
		__syncthreads();  // (the key groups have been read)
		mine[tid] = r;
		i8_cluster_sync();
		if (rank == 0) {
			float M = m_s[row];
#pragma unroll 1
			for (int p = 1; p < ks; p++) {
				const float pm = ac_remote(&m_s[row], p), pl = ac_remote(&l_s[row], p);
				if (pm == -INFINITY) continue;  // (no key of its chunks is visible)
				const float4 o4 = ac_remote4(&mine[tid], p);
				const float mn = fmaxf(M, pm), ea = M == -INFINITY ? 0.0f : expf(M - mn), eb = expf(pm - mn);
				L = fmaf(L, ea, pl * eb);
				r.x = fmaf(r.x, ea, o4.x * eb);
				r.y = fmaf(r.y, ea, o4.y * eb);
				r.z = fmaf(r.z, ea, o4.z * eb);
				r.w = fmaf(r.w, ea, o4.w * eb);
				M = mn;
			}
		}
		i8_cluster_sync();  // (nobody leaves while its memory is read)
		if (rank != 0) return;
	}
	r.x /= L;
	r.y /= L;
	r.z /= L;
	r.w /= L;
	const int s = s0 + qi;
	if (!x) {
		if (s < S) reinterpret_cast<float4 *>(o_out + (r0 + s) * 1024)[k4] = r;
		return;
	}
	const uint32_t mw = warp_umax(max(max(i8_abs_bits(r.x), i8_abs_bits(r.y)), max(i8_abs_bits(r.z), i8_abs_bits(r.w))));
	if (lane == 0) red[warp] = mw;
	__syncthreads();
	uint32_t mb = 0;
#pragma unroll
	for (int w = 0; w < 8; w++) mb = max(mb, red[qi * 8 + w]);
	if (s < S) {
		if (k4 == 0) rowscale[r0 + s] = i8_row_scale(mb);
		i8_pack4(x, groups, int(r0) + s, k4, r, i8_row_mul(mb));
	}
}

}  // namespace tg
