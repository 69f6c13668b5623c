// How the persistent decode kernel cuts a weight matrix into units, one per CTA, and a unit into tensor-core tiles. Plain C++
// without a CUDA type, so that the host compiler can walk a plan as the kernel does (tests/persist_plan_check.cpp).
#pragma once
#include <algorithm>
#include <vector>

#include "gemm_i8_tiles.h"  // TG_HOST_DEVICE

namespace tg {

constexpr int PS_THREADS = 384;
constexpr int PS_NW = PS_THREADS / 32;
constexpr int PS_TILES = 3;   // most MMA tiles of a unit: one per group of four warps
constexpr int PS_XCH = 144;   // bytes from one 16-byte chunk of the digits to the next: 8 rows of 16 bytes and 16 that keep the banks apart

// A unit is ncol columns of each of nmat matrices (up and gate together), 4 * nq rows. Column c (up columns, then gate
// columns) of K-segment s is row s * rows + c of `tiles` MMA tiles of mt rows; a tile's bytes are [16 k][mt rows / 8][8 rows][16 k],
// K-major core matrices of 128 bytes. Digit d of segment s is row 4 s + d of the other operand.
struct PsPhase {
	int ncol, nmat, nq;
	int nsplit;  // K-splits across CTAs
	int ntiles;  // column tiles
	int units;   // ntiles * nsplit
	int bytes;   // bytes of a unit: weights, then the scales of its columns
	int cta0;    // CTA of unit 0
	int rows;    // nmat * ncol
	int segs, mt, tiles;
	int steps;   // MMAs of a tile, 32 k each
	int seg_q;   // quads of a segment
	unsigned seg_mul;  // q / seg_q = q * seg_mul >> 20
	int x_sbo;   // bytes from the digits of two segments to those of the next two
	int x_bytes;
	int off_x, off_acc;  // digits and column sums in shared memory
};

// ------------------------------------------------------------------ addresses
// byte of (column c, 16-k chunk ch of segment seg) in a unit; 16 consecutive k follow, columns c + 1 .. of the same 8 rows 16 bytes apart
TG_HOST_DEVICE int ps_unit_offset(const PsPhase &ph, int c, int seg, int ch) {
	const int r = seg * ph.rows + c, t = r / ph.mt, m = r - t * ph.mt;
	return t * ph.mt * ph.seg_q * 4 + ch * ph.mt * 16 + (m / 8) * 128 + (m % 8) * 16;
}
// byte of digit 0 of quad q; the other digits follow 16 bytes apart
TG_HOST_DEVICE int ps_digit_offset(unsigned seg_mul, int seg_q, int sbo, int q) {
	const int seg = int((unsigned(q) * seg_mul) >> 20), kq = q - seg * seg_q;
	return (seg >> 1) * sbo + (seg & 1) * 64 + (kq >> 2) * PS_XCH + (kq & 3) * 4;
}
// first segment (even) whose digits the 16 columns of tile t's MMAs hold
TG_HOST_DEVICE int ps_tile_segment(int rows, int mt, int t) { return ((t * mt) / rows) & ~1; }
// warp w of tile t = w / 4 reads mt / 4 rows of one segment back: row r0 (entry of the column sums) from digit column `col` on
TG_HOST_DEVICE void ps_warp_rows(const PsPhase &ph, int w, int &r0, int &col) {
	const int t = w >> 2;
	r0 = t * ph.mt + (w & 3) * (ph.mt / 4);
	col = 4 * (r0 / ph.rows - ps_tile_segment(ph.rows, ph.mt, t));
}

// ------------------------------------------------------------------ plan
// MMA tiles of a unit of `rows` columns (of all its matrices) x 4 * nq rows: K-segments (a multiple of 32 k each) as
// further rows until they fill tiles of 64 or 128, at most one tile per group of four warps. A warp's 16 or 32 rows must lie in one
// segment, and a tile's segments within the four that its 16 digit columns hold. Returns the clocks from the digits to the
// column sums (measured: 430 + 23 per MMA of 64 rows, 38 per one of 128; a single issuing warp needs 33 and 39; 12 per segment to
// add), or a negative number.
inline double ps_mma_plan(PsPhase *ph) {
	double best = -1.0;
	const int K = 4 * ph->nq;
	for (int mt : {64, 128}) {
		if (ph->rows % (mt / 4)) continue;
		for (int segs = 1; segs <= K / 32; segs++) {
			if (K % (32 * segs) || (ph->rows * segs) % mt) continue;
			const int tiles = ph->rows * segs / mt, steps = K / segs / 32, seg_q = ph->nq / segs;
			if (tiles > PS_TILES) continue;
			int groups = (segs + 1) / 2;  // pairs of segments whose digits an MMA may read
			bool ok = true;
			for (int t = 0; t < tiles; t++) {
				const int start = ps_tile_segment(ph->rows, mt, t), last = ((t + 1) * mt - 1) / ph->rows;
				ok = ok && last - start < 4;
				groups = std::max(groups, start / 2 + 2);
			}
			const unsigned mul = unsigned(((1 << 20) + seg_q - 1) / seg_q);
			for (int q = 0; q < ph->nq; q++) ok = ok && int((unsigned(q) * mul) >> 20) == q / seg_q;
			if (!ok) continue;
			const double clk = 430.0 + tiles * steps * (tiles > 1 ? (mt == 64 ? 23.0 : 38.0) : (mt == 64 ? 33.0 : 39.0)) + 12.0 * segs;
			if (best < 0 || clk < best) {
				best = clk;
				ph->segs = segs;
				ph->mt = mt;
				ph->tiles = tiles;
				ph->steps = steps;
				ph->seg_q = seg_q;
				ph->seg_mul = mul;
				ph->x_sbo = seg_q / 4 * PS_XCH;
				ph->x_bytes = groups * ph->x_sbo;
			}
		}
	}
	return best;
}

// Plan of one matrix of K rows and nmat * N columns for G CTAs: columns per unit and K-splits across CTAs by an estimate of the
// phase's time in clocks: the product plus the bytes the phase makes CTAs poll (measured: about 76 clk per KB and CTA;
// `poll_kb(nsplit)` gives those KB for a split). col_blocks: a tile never straddles a multiple of these.
template <class F>
bool ps_plan(PsPhase *out, int K, int N, int nmat, int G, int max_bytes, const std::vector<int> &splits, const std::vector<int> &col_blocks, int max_nq, F poll_kb) {
	double best = 1e30;
	for (int ns : splits) {
		if ((K / 4) % ns) continue;
		const int nq = K / 4 / ns;
		if (nq > max_nq || nq % 8) continue;
		for (int ncol = 16; ncol <= PS_THREADS && ncol <= N; ncol += 16) {
			bool ok = N % ncol == 0;
			for (int cb : col_blocks) ok = ok && cb % ncol == 0;
			if (!ok) continue;
			PsPhase ph{};
			ph.ncol = ncol;
			ph.nmat = nmat;
			ph.rows = nmat * ncol;
			ph.nq = nq;
			ph.nsplit = ns;
			ph.ntiles = N / ncol;
			ph.units = ph.ntiles * ns;
			ph.bytes = ph.rows * nq * 4 + ph.rows * 4;
			if (ph.units > G || ph.bytes > max_bytes) continue;
			const double clk = ps_mma_plan(&ph);
			if (clk < 0) continue;
			// (a CTA without a unit is 4 clk worse: larger units elsewhere, and for the down projection a presence word to poll)
			const double cost = clk + 76.0 * poll_kb(ns) + 4.0 * (G - ph.units);
			if (cost < best) {
				best = cost;
				*out = ph;
			}
		}
	}
	return best < 1e30;
}

}  // namespace tg
