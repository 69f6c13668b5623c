// How the integer tensor-core GEMM cuts its work: the plan of a launch (CTAs per tile, tokens per tile, K-split) and the
// walk from a tile index to what the tile covers. Plain C++ without a CUDA type, so that the host compiler can walk
// every tile of a plan as the kernel does (tests/gemm_i8_tiles_check.cpp).
#pragma once
#include <algorithm>
#include <climits>
#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define TG_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define TG_HOST_DEVICE inline
#endif

namespace tg {

constexpr int I8_BK = 64;                      // k per block of the packed digits
constexpr int I8_GROUP_BYTES = 4 * 8 * I8_BK;  // one (K-block, token group): 4 digits x 8 tokens x 64 k
constexpr int I8_SK = 128;                     // k per stage
constexpr int I8_TG = 8;                       // token groups of a tile, at most
constexpr int I8_W_BYTES = 128 * I8_SK;

inline int i8_groups(int M) { return (M + 7) / 8; }

// ------------------------------------------------------------------ plan
// Tokens per tile, K-split and CTAs per tile of one GEMM launch, by an estimate in clocks of an SM: rounds of tiles per
// CTA (or pair) x (stages x the slowest of MMAs, operand bytes and the issuing threads + what a tile change costs) + what
// the consumer of the partial sums reads. The constants rank 2278 measured (shape, tile, split) combinations at 1 to 4001
// rows of all layer shapes: the choice is within 1 % of the best one on average. An MMA of N columns takes max(N / 2, 64) clk
// (a single CTA's are slowed to 1.28 of that by its operands' arrival), 78 B/clk arrive per SM with all SMs loading.
struct I8Plan {
	int cg, tg, tok_tiles, col_tiles, nsplit;
};
// N[0 .. ng): columns of the matrices of the launch; want_cg, want_split: nonzero asks for a choice (experiments). Raw sums that
// do not fit partial_floats even unsplit have no plan: the caller refuses them.
inline I8Plan i8_plan(int M, int K, int ng, const int *N, int num_sms, size_t partial_floats, int max_split, bool raw, int want_cg = 0, int want_split = 0) {
	I8Plan best{1, 1, 1, 1, 1};
	double best_cost = 1e30;
	const int groups = i8_groups(M), stages = K / I8_SK;
	int ntot = 0;
	for (int g = 0; g < ng; g++) ntot += N[g];
	for (int cg = 1; cg <= 2; cg++) {
		if (want_cg && cg != want_cg) continue;
		// up to 64 tokens the digits that a pair would share are little beside the weights (vocabulary matrix, pairs / single CTAs with the same
		// large stages, ncu: 640 rows, 3 tokens 44.2 / 36.0 us, 64 59.2 / 45.4; 1152 rows 58.0 / 58.8 and 72.0 / 71.0, but 256 tokens 200 / 227)
		if (!want_cg && cg == 2 && groups <= I8_TG) continue;
		int col_tiles = 0;
		for (int g = 0; g < ng; g++) col_tiles += (N[g] + 128 * cg - 1) / (128 * cg);
		const int workers = num_sms / cg;
		for (int tg = std::min(groups, I8_TG); tg >= std::max(1, std::min(groups, I8_TG) - 3); tg--) {
			const int tok_tiles = (groups + tg - 1) / tg;
			const double mma = 4.0 * std::max(16.0 * tg, 64.0) * (cg == 1 ? 1.28 : 1.0), in = I8_W_BYTES + 2.0 * tg * I8_GROUP_BYTES / cg;
			const double per_stage = std::max(std::max(mma, in / 78.0), 256.0);
			for (int ns = 1; ns <= std::min(max_split, stages); ns++) {
				if (want_split && ns != std::min(want_split, std::min(max_split, stages))) continue;
				if ((ns > 1 || raw) && size_t(ns) * M * ntot > partial_floats) break;
				const long tiles = long(tok_tiles) * col_tiles * ns, rounds = (tiles + workers - 1) / workers;
				double cost = double(rounds) * ((stages + ns - 1) / ns * per_stage + 2500.0) + tg * 100.0 + (cg - 1) * 4000.0;
				cost += double(raw ? ns - 1 : (ns > 1 ? ns + 1 : 0)) * M * ntot * 4.0 / 2500.0;  // partial sums read again, 2.5 KB a clock
				cost += raw ? (ns + 7) / 8 * 600.0 : (ns > 1 ? 4000.0 : 0.0);  // its dependent round trips; a launch more
				if (cost < best_cost) {
					best_cost = cost;
					best = I8Plan{cg, tg, tok_tiles, col_tiles, ns};
				}
			}
		}
	}
	if (best_cost == 1e30 && (want_cg || want_split)) return i8_plan(M, K, ng, N, num_sms, partial_floats, max_split, raw);
	return best;
}

// ------------------------------------------------------------------ walk
// x / d as a multiplication, exact for every 0 <= x < 2^31 (every role of a CTA computes its tiles between other things, and
// an integer division takes a single thread ~200 clk). With 2^s < d <= 2^(s+1) and m = ceil(2^(32+s) / d) < 2^32, m * d exceeds
// 2^(32+s) by less than d, which times x is below 2^(32+s): too little to reach the next quotient. (s = 0 is exact for x * d < 2^32
// only: the last of 70656 tiles, 4360 rows of the vocabulary matrix, came out as the first one of a K-split that does not exist.)
struct I8Div {
	int d;
	unsigned m;  // 0: d = 1
	int s;
};
inline I8Div i8_divisor(int d) {
	int s = 0;
	while ((1ll << (s + 1)) < d) s++;
	return I8Div{d, d <= 1 ? 0u : unsigned(((1ull << (32 + s)) + d - 1) / d), s};
}
TG_HOST_DEVICE int i8_div(int x, const I8Div &v) {
	if (v.m == 0) return x;
#ifdef __CUDA_ARCH__
	return int(__umulhi(unsigned(x), v.m) >> v.s);
#else
	return int(unsigned((uint64_t(unsigned(x)) * v.m) >> 32) >> v.s);
#endif
}

// Up to three weight matrices with the same K share one launch (q|k|v, up|gate): matrix g owns the column tiles
// [tile_end[g-1], tile_end[g])
struct I8Walk {
	int groups;         // token groups in the packed operand
	int tg, tok_tiles;  // token groups per tile, token tiles
	int n_fast;         // 1: consecutive tiles are the column tiles of one token tile; 0: the token tiles of one column tile
	int tiles;          // column tiles * tok_tiles * K-splits
	I8Div per_split;    // column tiles * tok_tiles
	I8Div fast;         // range of the faster tile index
	I8Div nsplit;
	int tile_end[3];    // (of unused slots INT_MAX)
	int K;
};

// tile index -> what it covers (every role of a CTA walks the same tiles)
struct I8Tile {
	int grp, n0;         // matrix, first column inside it
	int g0, ng;          // token groups
	int split, s0, ns;   // K-split, its first stage and number of stages
};
template <int CG> TG_HOST_DEVICE I8Tile i8_tile(const I8Walk &a, int t) {
	I8Tile r;
	r.split = i8_div(t, a.per_split);
	t -= r.split * a.per_split.d;
	const int hi = i8_div(t, a.fast), lo = t - hi * a.fast.d;
	const int ct = a.n_fast ? lo : hi, tt = a.n_fast ? hi : lo;
	r.grp = (ct >= a.tile_end[0]) + (ct >= a.tile_end[1]);
	// (selects over constant indices: a run-time index into the parameter arrays would move them to local memory)
	r.n0 = (ct - (r.grp == 0 ? 0 : (r.grp == 1 ? a.tile_end[0] : a.tile_end[1]))) * (128 * CG);
	r.g0 = tt * a.tg;
	r.ng = a.groups - r.g0 < a.tg ? a.groups - r.g0 : a.tg;
	const int all = a.K / I8_SK;
	r.s0 = i8_div(r.split * all, a.nsplit);
	r.ns = i8_div((r.split + 1) * all, a.nsplit) - r.s0;
	return r;
}

// the walk over M rows of a plan (its token tiles and K-split are the plan's)
inline void i8_fill_walk(I8Walk &a, const I8Plan &pl, int M, int K, int ng, const int *N) {
	int ntot = 0, tiles = 0;
	for (int g = 0; g < 3; g++) {
		if (g < ng) {
			ntot += N[g];
			tiles += (N[g] + 128 * pl.cg - 1) / (128 * pl.cg);
		}
		a.tile_end[g] = g < ng ? tiles : INT_MAX;
	}
	a.groups = i8_groups(M);
	a.tg = pl.tg;
	a.tok_tiles = pl.tok_tiles;
	a.tiles = pl.tok_tiles * pl.col_tiles * pl.nsplit;
	// matrices that stay in the L2 are swept once per token tile; the vocabulary matrix is read once for all token tiles
	a.n_fast = size_t(ntot) * K <= (size_t(48) << 20);
	a.per_split = i8_divisor(pl.col_tiles * pl.tok_tiles);
	a.fast = i8_divisor(a.n_fast ? pl.col_tiles : pl.tok_tiles);
	a.nsplit = i8_divisor(pl.nsplit);
	a.K = K;
}

}  // namespace tg
