// Multiplies units of the persistent decode kernel's plans with the kernel's own index arithmetic (persist_plan.h): weights and
// digits laid out by its address functions, MMAs read as the hardware reads them (core matrices of 8 rows x 16 bytes), sums read
// back per warp; compared with the product itself. Arguments: K N pairs (N columns of one matrix). Prints the number of units, or
// the first wrong one.
#include "../tiny-gemma_b200/csrc/persist_plan.h"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <cstdint>

using namespace tg;

static uint32_t g_seed = 1;
static uint32_t rnd() { return g_seed = g_seed * 1664525u + 1013904223u, g_seed >> 8; }

static bool unit_ok(const PsPhase &ph) {
	const int K = 4 * ph.nq, ks = K / ph.segs;
	const size_t weights = size_t(ph.rows) * K;
	if (size_t(ph.bytes) != weights + 4 * ph.rows || ph.bytes % 16) return false;  // (the columns' scales follow)
	std::vector<int8_t> W(weights), unit(weights), x(size_t(ph.x_bytes));
	std::vector<char> seen(weights, 0);
	std::vector<int32_t> v(K);
	for (auto &w : W) w = int8_t(int(rnd() % 255) - 127);
	for (auto &b : x) b = int8_t(rnd());  // (what no digit is written to must not count)
	for (auto &q : v) q = int32_t(rnd() * 128u + rnd() % 128u) % (1 << 30) * (rnd() & 1 ? 1 : -1);
	v[0] = 1 << 30;
	v[K - 1] = -(1 << 30);
	for (int c = 0; c < ph.rows; c++)
		for (int k = 0; k < K; k++) {
			const int seg = k / ks, o = ps_unit_offset(ph, c, seg, k % ks / 16) + k % 16;
			if (o < 0 || size_t(o) >= weights || seen[o]) return false;
			if (c % 4 == 0 && ps_unit_offset(ph, c + 3, seg, k % ks / 16) != o - k % 16 + 48) return false;  // (4 columns are stored together)
			seen[o] = 1;
			unit[o] = W[size_t(k) * ph.rows + c];
		}
	for (int q = 0; q < ph.nq; q++) {
		const int o = ps_digit_offset(ph.seg_mul, ph.seg_q, ph.x_sbo, q);
		if (o < 0 || o + 52 > ph.x_bytes) return false;
		for (int j = 0; j < 4; j++) {
			const uint32_t d = (uint32_t(v[4 * q + j]) + 0x80808080u) ^ 0x80808080u;
			for (int i = 0; i < 4; i++) x[o + 16 * i + j] = int8_t(d >> (8 * i));
		}
	}
	if (ph.tiles > PS_TILES || ph.rows * ph.segs != ph.tiles * ph.mt || ph.steps * 32 != ks || (ph.mt != 64 && ph.mt != 128)) return false;
	std::vector<int64_t> sum(size_t(ph.rows) * 4, 0);
	std::vector<char> read(size_t(ph.rows) * ph.segs, 0);
	for (int t = 0; t < ph.tiles; t++) {
		std::vector<int64_t> D(size_t(ph.mt) * 16, 0);
		const int a0 = t * ph.steps * ph.mt * 32, x0 = ps_tile_segment(ph.rows, ph.mt, t) / 2 * ph.x_sbo;
		for (int i = 0; i < ph.steps; i++)
			for (int m = 0; m < ph.mt; m++)
				for (int n = 0; n < 16; n++)
					for (int k = 0; k < 32; k++) {
						const int ao = a0 + i * ph.mt * 32 + (k / 16) * ph.mt * 16 + (m / 8) * 128 + (m % 8) * 16 + k % 16;
						const int xo = x0 + i * 2 * PS_XCH + (k / 16) * PS_XCH + (n / 8) * ph.x_sbo + (n % 8) * 16 + k % 16;
						if (size_t(ao) >= weights || xo >= ph.x_bytes) return false;
						D[m * 16 + n] += int(unit[ao]) * int(x[xo]);
					}
		for (int w = 4 * t; w < 4 * t + 4; w++) {
			int r0, col;
			ps_warp_rows(ph, w, r0, col);
			if (col < 0 || col > 12 || r0 / ph.rows != (r0 + ph.mt / 4 - 1) / ph.rows) return false;
			for (int l = 0; l < ph.mt / 4; l++) {
				if (read[r0 + l]++) return false;
				for (int i = 0; i < 4; i++) {
					const int64_t d = D[(size_t(w & 3) * (ph.mt / 4) + l) * 16 + col + i];
					if (d > INT32_MAX || d < INT32_MIN) return false;
					sum[size_t((r0 + l) % ph.rows) * 4 + i] += d;
				}
			}
		}
	}
	for (int c = 0; c < ph.rows; c++) {
		int64_t want = 0, got = 0;
		for (int k = 0; k < K; k++) want += int64_t(W[size_t(k) * ph.rows + c]) * v[k];
		for (int i = 3; i >= 0; i--) {
			if (sum[c * 4 + i] > INT32_MAX || sum[c * 4 + i] < INT32_MIN) return false;
			got = got * 256 + sum[c * 4 + i];
		}
		if (got != want) return false;
	}
	return true;
}

int main(int argc, char **argv) {
	int n = 0;
	auto run = [&](const PsPhase &ph, const char *what) {
		n++;
		if (unit_ok(ph)) return;
		printf("%s: %d x %d columns, %d rows, %d segments, %d tiles of %d\n", what, ph.nmat, ph.ncol, 4 * ph.nq, ph.segs, ph.tiles, ph.mt);
		exit(1);
	};
	// every unit shape that has a plan, up to 128 columns x 1152 rows
	for (int nmat = 1; nmat <= 2; nmat++)
		for (int ncol = 16; ncol * nmat <= 128; ncol += 16)
			for (int nq = 8; nq <= 288; nq += 8) {
				PsPhase ph{};
				ph.ncol = ncol;
				ph.nmat = nmat;
				ph.rows = nmat * ncol;
				ph.nq = nq;
				ph.bytes = ph.rows * nq * 4 + ph.rows * 4;
				if (ps_mma_plan(&ph) >= 0) run(ph, "shape");
			}
	for (int i = 1; i + 1 < argc; i += 2)
		for (int nmat = 1; nmat <= 2; nmat++)
			for (int G : {132, 148}) {
				PsPhase ph{};
				if (ps_plan(&ph, atoi(argv[i]), atoi(argv[i + 1]), nmat, G, 120 * 1024, nmat == 2 ? std::vector<int>{1} : std::vector<int>{1, 2, 3, 4}, {}, 1920,
				            [](int ns) { return 4.0 * ns; })) {
					if (ph.units > G || ph.ntiles * ph.ncol != atoi(argv[i + 1]) || 4 * ph.nq * ph.nsplit != atoi(argv[i])) return printf("plan\n"), 1;
					run(ph, "plan");
				}
			}
	printf("%d\n", n);
	return 0;
}
