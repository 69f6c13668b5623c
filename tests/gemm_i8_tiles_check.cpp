// Walks the tiles of the integer GEMM's plans with the kernel's own index arithmetic (gemm_i8_tiles.h) and compares every
// one with exact integer division. Arguments: K and N of every matrix size. Prints the number of tiles, or the first wrong one.
#include "../tiny-gemma_b200/csrc/gemm_i8_tiles.h"

#include <cstdio>
#include <cstdlib>
#include <vector>

using namespace tg;

static long long g_tiles = 0;

template <int CG> static bool same(const I8Walk &a, const int *cols, int ng, int t) {
	const long long x = t, cts = a.tile_end[ng - 1], nsplit = a.tiles / (cts * a.tok_tiles), per = cts * a.tok_tiles, in = x % per, all = a.K / I8_SK;
	const long long split = x / per, ct = a.n_fast ? in % cts : in / a.tok_tiles, tt = a.n_fast ? in / cts : in % a.tok_tiles;
	int grp = 0;
	long long first = 0;
	while (ct >= a.tile_end[grp]) first = a.tile_end[grp++];
	const long long n0 = (ct - first) * 128 * CG, g0 = tt * a.tg, s0 = split * all / nsplit, s1 = (split + 1) * all / nsplit;
	const long long ngr = a.groups - g0 < a.tg ? a.groups - g0 : a.tg;
	const I8Tile r = i8_tile<CG>(a, t);
	const bool in_range = r.split >= 0 && r.split < nsplit && r.grp < ng && r.n0 >= 0 && r.n0 < cols[r.grp] && r.g0 >= 0 && r.ng >= 1 &&
	                      r.g0 + r.ng <= a.groups && r.ns >= 1 && r.s0 >= 0 && r.s0 + r.ns <= all;
	g_tiles++;
	return in_range && r.split == split && r.grp == grp && r.n0 == n0 && r.g0 == g0 && r.ng == ngr && r.s0 == s0 && r.s0 + r.ns == s1;
}

// step 1 walks every tile; a larger one the tiles at both ends, at the ends of the splits and every step-th between them
static bool walk(int M, int K, int ng, const int *cols, size_t partial, bool raw, int cg, int split, int step) {
	int ntot = 0;
	for (int g = 0; g < ng; g++) ntot += cols[g];
	if (raw && size_t(M) * ntot > partial) return true;  // refused before it is launched
	const I8Plan pl = i8_plan(M, K, ng, cols, 148, partial, 16, raw, cg, split);
	I8Walk a{};
	i8_fill_walk(a, pl, M, K, ng, cols);
	const int per = a.tiles / pl.nsplit;
	for (int s = 0; s < pl.nsplit; s++)
		for (int i = 0; i < per; i = (step > 1 && i >= 64 && i + step < per - 64) ? i + step : i + 1) {
			const int t = s * per + i;
			if (!(pl.cg == 2 ? same<2>(a, cols, ng, t) : same<1>(a, cols, ng, t))) {
				std::printf("M %d K %d N %d (%d matrices): tile %d of %d is wrong (%d CTAs a tile, split %d)\n", M, K, cols[0], ng, t, a.tiles, pl.cg, pl.nsplit);
				return false;
			}
		}
	return true;
}

int main(int argc, char **argv) {
	std::vector<int> ks, ns;
	for (int i = 1; i < argc; i++) (ns.empty() && std::atoi(argv[i]) > 0 ? ks : ns).push_back(std::atoi(argv[i]));  // K .. 0 N ..
	const size_t partial = size_t(1) << 28;
	for (int K : ks)
		for (int N : ns) {
			if (N == 0) continue;
			const bool vocab = N > 100000;
			for (int M = 1; M <= 32768; M += M < 260 ? 1 : (vocab ? 1021 : 97))
				if (!walk(M, K, 1, &N, partial, false, 0, 0, vocab ? 61 : 1)) return 1;
			for (int M : {4353, 4360, 4361, 5000, 8192, 32768})
				for (int cg = 1; cg <= 2; cg++)
					if (!walk(M, K, 1, &N, partial, false, cg, 0, vocab ? 7 : 1)) return 1;
			for (int split : {2, 3, 5, 16})  // splits of every size, as far as the partial sums fit
				for (int M : {1, 63, 200, 1000, 4360})
					if (!walk(M, K, 1, &N, partial, true, 0, split, vocab ? 7 : 1)) return 1;
		}
	// the grouped launches: q|k|v and up|gate of both models
	const int sets[4][4] = {{640, 1024, 256, 256}, {1152, 1024, 256, 256}, {640, 2048, 2048, 0}, {1152, 6912, 6912, 0}};
	for (const int *s : sets)
		for (int M = 1; M <= 32768; M += M < 260 ? 1 : 211)
			if (!walk(M, s[0], s[3] ? 3 : 2, s + 1, partial, true, 0, 0, 1)) return 1;
	// the division itself up to the end of its range, at the multiples of the divisor and beside them
	for (long long d : {1ll, 2ll, 3ll, 7ll, 69ll, 1024ll, 2048ll, 60787ll, 65535ll, 65536ll, 65537ll, 70656ll, 1048573ll, 1073741825ll, 2147483647ll})
		for (long long k = 0; k <= 4000; k++)
			for (long long off = -1; off <= 1; off++)
				for (long long x : {k * d + off, (2147483647ll / d - k) * d + off})
					if (x >= 0 && x <= 2147483647ll && i8_div(int(x), i8_divisor(int(d))) != x / d) {
						std::printf("%lld / %lld is wrong\n", x, d);
						return 1;
					}
	std::printf("%lld tiles\n", g_tiles);
	return 0;
}
