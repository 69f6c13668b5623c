// Attention over fp32 K / V rows on the CUDA cores, for the shapes whose time is latency and memory traffic, not
// arithmetic: one decode step per sequence, and short prompts.
//
// The rows of a sequence's keys (values) follow each other in memory, so four of them are ONE bulk copy of 4 KB into a
// warp's ring in shared memory: the whole traffic of a CTA is asynchronous and costs no registers. Both kernels take a step of
// four keys against the heads of a query per warp: scores (a lane holds 8 of the 256 dimensions, and the lanes' partial sums meet in a
// reduce-scatter), a softmax step with a running maximum of the warp's own, the products with V. The warps' parts are joined at the end.
//
// The result leaves as the digits of the O projection's operand (kernels_gemm_i8.cuh) where the caller wants them: the
// CTA that finishes a row has all of it.
#pragma once
#include "kernels_decode.cuh"  // AT_NH, AT_HD
#include "kernels_gemm_i8.cuh"
#include "tg_common.cuh"

namespace tg {

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

__device__ __forceinline__ uint32_t ac_mapa(const void *p, int rank) {
	uint32_t r;
	asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
	return r;
}
// a wait ran out: report it, and give the copies in flight time to land before the shared memory goes to another use
__device__ __noinline__ void ac_give_up(int *err) {
	*static_cast<volatile int *>(err) = 6;
	const long long t0 = clock64();
	while (clock64() - t0 < 2000000) {
	}
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
	int nsplit, cluster;  // CTAs per sequence, and how many of them form a cluster (1: none)
	int polls;            // limit of a wait for copies
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
// Few sequences: the splits of a sequence are clusters of CTAs, whose parts meet in the first one's shared memory; only where a cache takes more than
// one cluster do parts go through memory and a ticket (a store, a fence, an atomic and a load, one behind the other: 1.5 us).
// Steps in us, through memory / in clusters. 1B: 2 sequences of 61 positions 778 / 732, 8 837 / 752, 8 of 1500 910 / 868, 4 and 8 of 6000 900 / 896 and 975 / 953;
// 270m: 451 / 411, 492 / 429, 531 / 501, 528 / 510 and 572 / 571; 16 of 61 501 / 487, but 16 of 500 539 / 589 (one CTA per SM): up to 8 sequences. (4 and 8 long
// caches come to 16 clusters; a GPU holds 15 or 16 at once, by which of its SMs are in use.)
constexpr int AD_CLUSTER = 8, AD_CLUSTER_SEQS = 8;
inline int attn_decode_smem(int cluster) { return AD_SMEM + (cluster - 1) * AT_PART * 4; }

__global__ void __launch_bounds__(AT_THREADS, 2) attn_decode_kernel(AttnArgs a) {
	extern __shared__ __align__(128) uint8_t ac_smem[];
	__shared__ __align__(16) float rowbuf[AT_NH * AT_HD + 2 * AT_HD];  // q | k | v of the new token, normed and rotated
	__shared__ float m_s[AT_THREADS / 32][AT_NH], l_s[AT_THREADS / 32][AT_NH];
	__shared__ uint64_t full[AT_THREADS / 32][AD_STAGES];
	__shared__ uint32_t red[AT_THREADS / 32];
	__shared__ int s_last;
	const int b = blockIdx.y, split = blockIdx.x, rank = a.cluster > 1 ? split % AD_CLUSTER : 0;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	pdl_trigger();
	uint8_t *ring = ac_smem + warp * (AD_STAGES * AD_BUF);
	if (lane == 0) {
		for (int i = 0; i < AD_STAGES; i++) mbar_init(&full[warp][i], 1);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	__syncwarp();
	if (a.cluster > 1) i8_cluster_sync();
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
	pdl_wait();
	int pos = a.step_pos[b];
	const int base = a.is_local ? a.ring_base[b] : 0;
	// the projections' K-splits, QB of them in flight together with the position; they are added behind the requests for the cache
	constexpr int QB = 10;
	const float4 *qkv = reinterpret_cast<const float4 *>(a.qkv + size_t(b) * NQ + warp * AT_HD) + lane;
	const size_t sstride = size_t(a.qkv_B) * (NQ / 4);
	const int nsp = warp < AT_NH + 2 ? max(a.qkv_nsplit, 1) : 0;
	float4 u[QB], v[QB];
#pragma unroll
	for (int q = 0; q < QB; q++) {
		u[q] = v[q] = z4;
		if (q < nsp) {
			u[q] = qkv[size_t(q) * sstride];
			v[q] = qkv[size_t(q) * sstride + 32];
		}
	}
	int valid = min(pos + 1, a.slots);
	if (!a.is_local && pos >= a.slots) {  // cache full: refuse to write out of bounds
		if (tid == 0) *a.err_flag = 2;
		pos = a.slots - 1;
	}
	// whole rounds of 32 keys are dealt out to the splits; splits without any leave at once
	const int rounds = (valid + AD_ROUND - 1) / AD_ROUND;
	int per = 1, nact = rounds;
	if (rounds > a.nsplit) {
		per = (rounds + a.nsplit - 1) / a.nsplit;
		nact = (rounds + per - 1) / per;
	}
	// The cluster's first CTA stays until every other one has handed over its part, has none or has given up: it waits at the cluster's barrier, which the
	// others reach because all waits in front of it are bounded. (A bounded wait of its own could run out first, and a part would arrive in a CTA that has left.)
	auto hand_over = [] {
		__syncwarp();
		asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
	};
	if (split >= nact) {
		if (a.cluster > 1) hand_over();
		return;
	}
	const int j0 = split * per * AD_ROUND, j1 = min(valid, j0 + per * AD_ROUND);
	const int jw = j0 + AD_KEYS * warp, nit = max(0, (j1 - jw + AD_ROUND - 1) / AD_ROUND);  // this warp's first key, its groups of keys
	float *kc = a.kcache + size_t(b) * a.slots * AT_HD, *vc = a.vcache + size_t(b) * a.slots * AT_HD;
	// Caches that no L2 holds until the next step are read evict-first: at normal priority they push out what the launches around them exchange (steps of 1B:
	// 256 sequences of 178 positions 2140 -> 2040 us, 128 of 300 1684 -> 1627). Smaller ones lose a little (16 of 500, 270m, 531 -> 535).
	const bool stream = long(gridDim.y) * valid > 16384;
	const uint64_t policy = l2_evict_first_policy();
	// item i of the warp's ring: the keys (i even) or the values (i odd) of group i / 2; called by the whole warp
	int items = 2 * nit;  // (none any more behind a wait that ran out: the stage's barrier may still count an older copy)
	auto issue = [&](int i) {
		const int j = jw + (i >> 1) * AD_ROUND, st = i % AD_STAGES;
		const uint32_t bytes = uint32_t(min(AD_KEYS, j1 - j)) * 1024u;
		if (tc_elect() && i < items) {
			mbar_expect_tx(&full[warp][st], bytes);
			const float *src = (i & 1 ? vc : kc) + size_t(j) * AT_HD;
			if (stream)
				asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(smem_u32(ring + st * AD_BUF)),
				             "l"(src), "r"(bytes), "r"(smem_u32(&full[warp][st])), "l"(policy)
				             : "memory");
			else
				bulk_load(ring + st * AD_BUF, src, bytes, &full[warp][st]);
		}
	};
#pragma unroll
	for (int i = 0; i < AD_STAGES; i++) issue(i);
	const int slot = a.is_local ? (pos - base) % a.slots : pos;
	float4 lo = z4, hi = z4, c0 = z4, c1 = z4, n0 = z4, n1 = z4;
	if (warp <= AT_NH) {
		const float4 *cr = reinterpret_cast<const float4 *>(a.cosT + size_t(pos) * AT_HD), *sr = reinterpret_cast<const float4 *>(a.sinT + size_t(pos) * AT_HD);
		c0 = cr[lane];
		c1 = cr[32 + lane];
		n0 = sr[lane];
		n1 = sr[32 + lane];
	}
	auto add = [](float4 &x, const float4 &y) {
		x.x += y.x;
		x.y += y.y;
		x.z += y.z;
		x.w += y.w;
	};
#pragma unroll
	for (int q = 0; q < QB; q++) {
		add(lo, u[q]);
		add(hi, v[q]);
	}
	for (int q = QB; q < nsp; q++) {
		add(lo, qkv[size_t(q) * sstride]);
		add(hi, qkv[size_t(q) * sstride + 32]);
	}
	if (a.qkv_nsplit > 0) {
		lo = make_float4(lo.x * s0.x, lo.y * s0.y, lo.z * s0.z, lo.w * s0.w);
		hi = make_float4(hi.x * s1.x, hi.y * s1.y, hi.z * s1.z, hi.w * s1.w);
	}
	if (warp <= AT_NH) {  // per-head norm and RoPE; lane owns d = 4 lane .. and the partners 128 + d
		// the reference scales q by 1/sqrt(256) = 2^-4 before the dot products (ops.hpp:262,283)
		const float qs = warp < AT_NH ? 0.0625f : 1.0f;
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
	int cap = a.polls;
	auto wait = [&](int i) {
		tc_wait_cap(&full[warp][i % AD_STAGES], i / AD_STAGES & 1, cap);
		if (cap == 0) items = 0;
	};
	for (int it = 0; it < nit; it++) {
		const int j = jw + it * AD_ROUND, n = min(AD_KEYS, j1 - j);
		const int ik = 2 * it, iv = 2 * it + 1;
		uint8_t *K = ring + ik % AD_STAGES * AD_BUF, *V = ring + iv % AD_STAGES * AD_BUF;
		wait(ik);
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
		wait(iv);
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
	if (cap == 0) ac_give_up(a.err_flag);
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
	int nparts = nact, part = split;
	if (a.cluster > 1) {
		float *in = reinterpret_cast<float *>(ac_smem + AD_SMEM);  // the other CTAs' parts, laid out as in memory
		if (rank != 0) {
			const uint32_t dst = ac_mapa(in + (rank - 1) * AT_PART, 0);
			asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(dst + 16u * tid), "f"(r.x), "f"(r.y), "f"(r.z), "f"(r.w) : "memory");
			if (d4 == 0)
				asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(dst + 4u * (AT_NH * AT_HD) + 8u * h), "f"(Ms), "f"(L) : "memory");
			hand_over();
			return;
		}
		hand_over();
		asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
		const int n = min(AD_CLUSTER, nact - split);
#pragma unroll 1
		for (int p = 1; p < n; p++, in += AT_PART) {  // (every part has a key)
			const float4 o4 = reinterpret_cast<const float4 *>(in)[tid];
			const float2 ml = reinterpret_cast<const float2 *>(in + AT_NH * AT_HD)[h];
			const float mn = fmaxf(Ms, ml.x), ea = expf(Ms - mn), eb = expf(ml.x - mn);
			L = fmaf(L, ea, ml.y * eb);
			r = make_float4(r.x * ea, r.y * ea, r.z * ea, r.w * ea);
			ac_fma4(r, eb, o4);
			Ms = mn;
		}
		nparts = (nact + AD_CLUSTER - 1) / AD_CLUSTER;
		part = split / AD_CLUSTER;
	}
	if (nparts > 1) {
		float *pb = a.part + size_t(b) * a.nsplit * AT_PART;
		float *prow = pb + size_t(part) * AT_PART;
		__stcg(reinterpret_cast<float4 *>(prow) + tid, r);
		if (d4 == 0) {
			__stcg(prow + AT_NH * AT_HD + h, Ms);
			__stcg(prow + AT_NH * AT_HD + 4 + h, L);
		}
		__threadfence();
		__syncthreads();
		if (tid == 0) s_last = atomicAdd(&a.tickets[b], 1u) == unsigned(nparts - 1);
		__syncthreads();
		if (!s_last) return;
		__threadfence();
		constexpr int PB = 16;  // parts requested together (8: 300 positions of three sequences in 10 parts 0.6 us a layer slower)
		float M = -INFINITY;
		r = make_float4(0.f, 0.f, 0.f, 0.f);
		L = 0.0f;
		for (int s0 = 0; s0 < nparts; s0 += PB) {
			float4 v[PB];
			float ms[PB], ls[PB], mn = M;
#pragma unroll
			for (int q = 0; q < PB; q++) {
				v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
				ms[q] = -INFINITY;
				ls[q] = 0.0f;
				if (s0 + q < nparts) {
					const float *p = pb + size_t(s0 + q) * AT_PART;
					v[q] = __ldcg(reinterpret_cast<const float4 *>(p) + tid);
					ms[q] = __ldcg(p + AT_NH * AT_HD + h);
					ls[q] = __ldcg(p + AT_NH * AT_HD + 4 + h);
				}
			}
#pragma unroll
			for (int q = 0; q < PB; q++) mn = fmaxf(mn, ms[q]);
			const float c = expf(M - mn);  // (0 for the first parts)
			M = mn;
			L *= c;
			r = make_float4(r.x * c, r.y * c, r.z * c, r.w * c);
#pragma unroll
			for (int q = 0; q < PB; q++) {
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
// Two queries (8 rows of 4 heads) per CTA of 16 warps. As in the decode kernel a warp takes 4 keys at a time against the four heads of
// one query, with a running maximum of its own; warps g and g + 8 share the keys of group g, which arrive through a ring of the group.
// Nothing in the walk waits for another group. Shared memory and shuffles (~1500 clk per 32 keys and two queries), FMAs (1100) and copies (64 KB) bound it.
// q [S][1024], k and v [off + S][256] per prompt; blockIdx.y is the
// prompt. Query s is the token at key off + s (off > 0: a continuation, its context comes first). Causal; on local layers
// a query sees at most `window` keys before itself (the reference's prefill rule, ops.hpp:439-443).
// The CTAs of a cluster share the keys of two queries, and hand their parts to the first one, which joins them in order; where two queries have
// so few keys that one CTA takes no longer for them than a share of the longest walk, every CTA of a cluster takes two queries of its own.
// 178 tokens, the longest walk of a launch: 10.2 us with 32 keys at a time for all 16 warps between three barriers, 8.0 now, and no
// second wave of CTAs (all walks shared by two: 178 CTAs).
constexpr int APS_GROUPS = 8, APS_THREADS = 2 * 32 * APS_GROUPS;
constexpr int APS_KEYS = 4, APS_STAGES = 3;  // keys of a step; K and V of so many steps in a group's ring
constexpr int APS_BUF = APS_KEYS * 1024;
constexpr int APS_RING = APS_GROUPS * APS_STAGES * 2 * APS_BUF;
constexpr int APS_PART = 2 * AT_NH * AT_HD + 2 * 2 * AT_NH;  // floats that a CTA hands over: 8 rows, their maxima and sums
constexpr int APS_MAX_KS = 5;                                // CTAs of a cluster (their parts lie beside the ring)
// ks: CTAs of a cluster. shared: the clusters that share two queries each, those with the most keys
struct AttnSmallPlan {
	int ks, shared, clusters;
	int smem() const { return APS_RING + (ks - 1) * APS_PART * 4; }
};
// For a prompt of S tokens behind `off` others. By the prompt alone: a prompt of a group gets the bits that it gets by itself. The largest cluster
// with two rounds of 32 keys per CTA at least (one where there are three in all: 61 tokens of 1B 1139 -> 1125 us, but 128 1283 -> 1297) whose CTAs are all resident at once (one per SM; the SMs of a GPC hold whole clusters): 178 tokens 2, 61 behind 1500 cached ones 4. How many
// that are differs by GPU (clusters of 3, 4 and 5: 135 to 138, 128 to 132 and 115 to 130 CTAs seen); as constants, or a prompt's bits would differ with it.
inline AttnSmallPlan attn_small_plan(int S, int off, int is_local, int window) {
	constexpr int ROUND = APS_GROUPS * APS_KEYS, resident[APS_MAX_KS + 1] = {0, 148, 148, 138, 128, 115};
	const int pairs = (S + 1) / 2, most = is_local ? std::min(off + S, window + 2) : off + S;
	const int rounds = (most + ROUND - 1) / ROUND;
	for (int ks = std::min(APS_MAX_KS, rounds <= 3 ? rounds : rounds / 2); ks > 1; ks--) {
		const int share = (most + ks * ROUND - 1) / (ks * ROUND) * ROUND;                // keys of a CTA of the longest walk
		const int alone = most <= share ? pairs : std::min(pairs, std::max(0, share - off) / 2);  // pair i has off + 2 i + 2 keys
		const int clusters = pairs - alone + (alone + ks - 1) / ks;
		if (clusters * ks <= resident[ks]) return AttnSmallPlan{ks, pairs - alone, clusters};
	}
	return AttnSmallPlan{1, 0, pairs};
}
__global__ void __launch_bounds__(APS_THREADS, 1) attn_prefill_small_kernel(float *o_out, uint8_t *x, float *rowscale, int groups, const float *q,
                                                                            const float *k, const float *v, int S, int off, int is_local, int window,
                                                                            int cluster, int shared, int polls, int *err) {
	extern __shared__ __align__(128) uint8_t ac_smem[];
	constexpr int R = 2 * AT_NH, H = AT_NH;  // query rows: query * 4 + head
	__shared__ float m_s[APS_GROUPS][R], l_s[APS_GROUPS][R];
	__shared__ uint64_t full[APS_GROUPS][APS_STAGES], done[APS_GROUPS][APS_STAGES];  // a step's keys and values landed; both warps have read them
	__shared__ uint32_t red[APS_THREADS / 32];
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, grp = warp & (APS_GROUPS - 1), qi = warp / APS_GROUPS;  // this warp's query
	uint8_t *ring = ac_smem + grp * (APS_STAGES * 2 * APS_BUF);
	if (tid < APS_GROUPS * APS_STAGES) {
		mbar_init(&full[0][0] + tid, 1);
		mbar_init(&done[0][0] + tid, 2);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	__syncthreads();
	if (cluster > 1) asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");  // (waited for before anything is handed over)
	pdl_trigger();
	pdl_wait();
	const size_t r0 = size_t(blockIdx.y) * S;
	// the cluster's queries (the longest walks start first), among how many CTAs they are shared, and which of them this one is
	const int c = int(blockIdx.x) / cluster, last = (S + 1) / 2 - 1;
	const int ks = c < shared ? cluster : 1, rank = ks > 1 ? int(blockIdx.x) % cluster : 0;
	const int pair = last - (c < shared ? c : shared + (c - shared) * cluster + int(blockIdx.x) % cluster), s0 = 2 * max(pair, 0);
	const int s_last = min(S - 1, s0 + 1);
	const int j0 = (is_local && off + s0 >= window) ? off + s0 - window : 0, j1 = off + s_last + 1;
	// steps of four keys are dealt out to all groups of the cluster in turn: this group's first key, the distance to its next, how many steps
	const int jw = j0 + APS_KEYS * (rank * APS_GROUPS + grp), jd = APS_KEYS * APS_GROUPS * ks, nit = pair < 0 ? 0 : max(0, (j1 - jw + jd - 1) / jd);
	k += r0 * 256;  // (a continuation is one sequence: r0 = 0)
	v += r0 * 256;
	auto issue = [&](int i, int cap) {  // step i of the group; called by the whole warp (cap = 0: not behind a wait that ran out)
		const int j = jw + i * jd, st = i % APS_STAGES;
		if (i < nit && tc_elect() && cap > 0) {
			const uint32_t bytes = uint32_t(min(APS_KEYS, j1 - j)) * 1024u;
			mbar_expect_tx(&full[grp][st], 2 * bytes);
			bulk_load(ring + st * 2 * APS_BUF, k + size_t(j) * 256, bytes, &full[grp][st]);
			bulk_load(ring + st * 2 * APS_BUF + APS_BUF, v + size_t(j) * 256, bytes, &full[grp][st]);
		}
	};
	if (qi == 0) {
#pragma unroll
		for (int i = 0; i < APS_STAGES; i++) issue(i, 1);
	}
	// A lane keeps the heads, and the keys of a step, in an order of its own for the scores (slot ^ hperm, slot ^ kperm): every round of the
	// reduce-scatter then keeps the lower and sends the upper slots, without selects.
	const int hperm = (lane >> 1) & 3, kperm = lane >> 3;
	const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
	float4 q0[H], q1[H], o0[H], o1[H];  // lane: dimensions 4 lane .. and 128 + 4 lane ..
	{
		// (a query past the prompt's end repeats the last one; it is not stored)
		const float4 *qr = reinterpret_cast<const float4 *>(q + (r0 + min(s0 + qi, S - 1)) * 1024) + lane;
#pragma unroll
		for (int h = 0; h < H; h++) {
			q0[h] = qr[(h ^ hperm) * 64];
			q1[h] = qr[(h ^ hperm) * 64 + 32];
			o0[h] = o1[h] = z4;
		}
	}
#pragma unroll
	for (int h = 0; h < H; h++) {  // exact: the reference scales q by 1/sqrt(256) = 2^-4 before the dot products
		q0[h].x *= 0.0625f; q0[h].y *= 0.0625f; q0[h].z *= 0.0625f; q0[h].w *= 0.0625f;
		q1[h].x *= 0.0625f; q1[h].y *= 0.0625f; q1[h].z *= 0.0625f; q1[h].w *= 0.0625f;
	}
	float m = -INFINITY, l = 0.0f;  // of head hperm; this lane's score of a step is key kperm's
	const int mine = off + s0 + qi, first = is_local ? mine - window : 0;  // the query's own key, the first one that it sees
	int cap = polls;
	for (int it = 0; it < nit; it++) {
		const int j = jw + it * jd, n = min(APS_KEYS, j1 - j), st = it % APS_STAGES, ph = it / APS_STAGES & 1;
		const uint8_t *K = ring + st * 2 * APS_BUF, *V = K + APS_BUF;
		tc_wait_cap(&full[grp][st], ph, cap);
		float t[16];
#pragma unroll
		for (int kk = 0; kk < APS_KEYS; kk++) {  // (rows past n hold an older step's keys, or nothing yet: their scores are not used)
			const uint8_t *kr = K + (kk ^ kperm) * 1024 + 16 * lane;
			const float4 k0 = *reinterpret_cast<const float4 *>(kr), k1 = *reinterpret_cast<const float4 *>(kr + 512);
#pragma unroll
			for (int h = 0; h < H; h++) t[kk * H + h] = ac_dot8x2(q0[h], q1[h], k0, k1);
		}
		// the partner's lane differs in the bit that the round splits on: its upper slot is the key and head of this lane's lower one
#pragma unroll
		for (int o = 8; o >= 1; o >>= 1)
#pragma unroll
			for (int i = 0; i < o; i++) t[i] += __shfl_xor_sync(0xffffffffu, t[i + o], 2 * o);
		t[0] += __shfl_xor_sync(0xffffffffu, t[0], 1);
		const int key = j + kperm;
		const bool vis = kperm < n && key <= mine && key >= first;
		const float z = vis ? t[0] : -INFINITY;
		float mn = fmaxf(m, z);
		mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 8));
		mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 16));
		// (mn may still be -inf: no key is visible yet, since the window starts later or the step lies behind the query, or all four scores overflowed to it)
		const float p = z != -INFINITY ? expf(z - mn) : 0.0f, cr = m == mn ? 1.0f : expf(m - mn);
		float ps = p + __shfl_xor_sync(0xffffffffu, p, 8);
		ps += __shfl_xor_sync(0xffffffffu, ps, 16);
		l = fmaf(l, cr, ps);
		m = mn;
		if (__any_sync(0xffffffffu, cr != 1.0f)) {
#pragma unroll
			for (int h = 0; h < H; h++) {
				const float c = __shfl_sync(0xffffffffu, cr, 2 * h);
				o0[h] = make_float4(o0[h].x * c, o0[h].y * c, o0[h].z * c, o0[h].w * c);
				o1[h] = make_float4(o1[h].x * c, o1[h].y * c, o1[h].z * c, o1[h].w * c);
			}
		}
#pragma unroll
		for (int kk = 0; kk < APS_KEYS; kk++) {
			if (kk < n) {
				const float4 v0 = *reinterpret_cast<const float4 *>(V + kk * 1024 + 16 * lane), v1 = *reinterpret_cast<const float4 *>(V + kk * 1024 + 512 + 16 * lane);
#pragma unroll
				for (int h = 0; h < H; h++) {
					const float w = __shfl_sync(0xffffffffu, p, 8 * kk + 2 * h);
					ac_fma4x2(o0[h], w, v0);
					ac_fma4x2(o1[h], w, v1);
				}
			}
		}
		__syncwarp();
		if (it + APS_STAGES < nit) {
			if (lane == 0) mbar_arrive(&done[grp][st]);
			if (qi == 0) {  // (its other warp is about as far)
				tc_wait_cap(&done[grp][st], ph, cap);
				issue(it + APS_STAGES, cap);
			}
		}
	}
	if (cap == 0) ac_give_up(err);
	// ---- join the groups: thread (query, k4) ends up with four of its query's 1024 outputs
	__syncthreads();  // (every warp has read its ring)
	float4 *jb = reinterpret_cast<float4 *>(ac_smem);
#pragma unroll
	for (int h = 0; h < H; h++) {
		jb[(grp * R + qi * H + h) * 64 + lane] = o0[h];
		jb[(grp * R + qi * H + h) * 64 + 32 + lane] = o1[h];
	}
	if (lane < 2 * H && !(lane & 1)) {
		m_s[grp][qi * H + (lane >> 1)] = m;
		l_s[grp][qi * H + (lane >> 1)] = l;
	}
	__syncthreads();
	const int k4 = tid & 255, row = tid >> 6;  // (query tid / 256 is the warp's own)
	float M = -INFINITY, L = 0.0f;
#pragma unroll
	for (int g = 0; g < APS_GROUPS; g++) M = fmaxf(M, m_s[g][row]);
	float4 r = z4;
#pragma unroll
	for (int g = 0; g < APS_GROUPS; g++) {
		const float mg = m_s[g][row], w = mg == -INFINITY ? 0.0f : expf(mg - M);
		L = fmaf(l_s[g][row], w, L);
		ac_fma4(r, w, jb[(g * R + row) * 64 + (k4 & 63)]);
	}
	if (cluster > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
	if (pair < 0) return;
	if (ks > 1) {  // the other CTAs' parts lie behind the first one's ring, rows and then maxima and sums
		const float *in = reinterpret_cast<const float *>(ac_smem + APS_RING);
		if (rank != 0) {
			const uint32_t dst = ac_mapa(in + (rank - 1) * APS_PART, 0);
			asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(dst + 16u * tid), "f"(r.x), "f"(r.y), "f"(r.z), "f"(r.w) : "memory");
			if ((k4 & 63) == 0)
				asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(dst + 4u * (R * AT_HD) + 8u * row), "f"(M), "f"(L) : "memory");
		}
		asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
		if (rank != 0) return;
#pragma unroll 1
		for (int p = 0; p < ks - 1; p++, in += APS_PART) {
			const float4 o4 = reinterpret_cast<const float4 *>(in)[tid];
			const float2 ml = reinterpret_cast<const float2 *>(in + R * AT_HD)[row];
			const float mn = fmaxf(M, ml.x);
			if (mn == -INFINITY) continue;  // (no key of either is visible)
			const float ea = expf(M - mn), eb = expf(ml.x - mn);
			L = fmaf(L, ea, ml.y * eb);
			r.x = fmaf(r.x, ea, o4.x * eb);
			r.y = fmaf(r.y, ea, o4.y * eb);
			r.z = fmaf(r.z, ea, o4.z * eb);
			r.w = fmaf(r.w, ea, o4.w * eb);
			M = mn;
		}
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
