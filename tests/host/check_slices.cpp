// FP64 products by digit slices (ctg_slices.h) and their tile lists (lower_dot in ctg_plan.cpp), walked on
// the host as the kernel walks them: every output entry is covered once, every operand access lies in
// its block, the digit sums of 128 terms stay within 2^24 (exact in FP32), and a result differs from the
// sum in extended integers by at most its own rounding and the digits that the slices cut off.
// Built and run by tests/test_host_logic.py; no GPU involved.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "ctg_plan.h"
#include "ctg_slices.h"

namespace ctg {
int tc_tile_rows() { return 128; }
int tc_k_chunk(int) { return 32; }
}  // namespace ctg
using namespace ctg;

static uint64_t bits_of(double x)
{
	uint64_t b;
	memcpy(&b, &x, 8);
	return b;
}

static double value_of(uint64_t b)
{
	double x;
	memcpy(&x, &b, 8);
	return x;
}

static int bad = 0;

// one result from the digits of its two rows; returns the biased exponents of the rows
static double slice_dot(const std::vector<double>& x, const std::vector<double>& y, int& E, int& F)
{
	E = F = 0;
	for (double v : x) E = std::max(E, (int)((bits_of(v) >> 52) & 0x7ff));
	for (double v : y) F = std::max(F, (int)((bits_of(v) >> 52) & 0x7ff));
	int64_t hi = 0, lo = 0;
	for (size_t k0 = 0; k0 < x.size(); k0 += SLICE_K)
	{
		int64_t acc[SLICES] = {0};
		for (size_t k = k0; k < std::min(x.size(), k0 + SLICE_K); k++)
		{
			const uint64_t bx = bits_of(x[k]), by = bits_of(y[k]);
			const uint64_t u = slice_digits((uint32_t)(bx >> 32), (uint32_t)bx, std::max(E, SLICE_EXP_MIN));
			const uint64_t v = slice_digits((uint32_t)(by >> 32), (uint32_t)by, std::max(F, SLICE_EXP_MIN));
			for (int s = 0; s < SLICES; s++)
				for (int t = 0; s + t < SLICES; t++)
					acc[s + t] += ((int64_t)((u >> (56 - 8 * s)) & 255) - 128) * ((int64_t)((v >> (56 - 8 * t)) & 255) - 128) *
					              ((bx ^ by) >> 63 ? -1 : 1);
		}
		for (int o = 0; o < SLICES; o++)
		{
			// 128 terms below 2^24 (exact in FP32), the 32 of a short flush and the orders 0 .. 2 below 2^22
			if (std::llabs(acc[o]) >= (1 << 24) ||
			    ((o <= 2 || std::min(x.size(), k0 + SLICE_K) - k0 <= 32) && std::llabs(acc[o]) >= (1 << 22)))
				bad++;
			if (o < 4) hi += acc[o] * ((int64_t)1 << (24 - 8 * o));
			else lo += acc[o] * ((int64_t)1 << (56 - 8 * o));
		}
	}
	if (E == 0 || F == 0) return 0;
	if (!slice_in_range(slice_top(E, F))) bad++;
	return value_of(slice_value(hi, lo, slice_top(E, F)));
}

// sum x y to about 106 bits (products and sums with their rounding errors)
static double accurate_dot(const std::vector<double>& x, const std::vector<double>& y)
{
	double s = 0, c = 0;
	for (size_t k = 0; k < x.size(); k++)
	{
		const double p = x[k] * y[k], e = std::fma(x[k], y[k], -p);
		const double t = s + p, z = t - s;
		c += (s - (t - z)) + (p - z) + e;
		s = t;
	}
	return s + c;
}

int main()
{
	setenv("CTGPU_SLICE_GEMM", "1", 1);
	std::mt19937 rng(11);
	std::normal_distribution<double> nd;
	// digits: balanced, and together the number to 2^-62 of the row's power of two
	for (int t = 0; t < 20000; t++)
	{
		const double x = std::ldexp(nd(rng), (int)(rng() % 80) - 40);
		const int E = (int)((bits_of(x) >> 52) & 0x7ff) + (int)(rng() % 70);
		const uint64_t u = slice_digits((uint32_t)(bits_of(x) >> 32), (uint32_t)bits_of(x), E);
		__int128 v = 0;
		for (int s = 0; s < SLICES; s++) v = v * 256 + ((int)((u >> (56 - 8 * s)) & 255) - 128);
		const double back = std::copysign(std::ldexp((double)(int64_t)v, E - 1022 - 62), x);
		if (std::fabs(back - x) > std::ldexp(1.0, E - 1022 - 62)) bad++;
		if (E - (int)((bits_of(x) >> 52) & 0x7ff) <= 9 && back != x) bad++;
	}
	// results: random rows, graded rows, cancelling rows, rows of zeros, extreme digits
	for (int t = 0; t < 3000; t++)
	{
		const size_t k = 1 + rng() % 700;
		std::vector<double> x(k), y(k);
		const int kind = t % 5;
		for (size_t i = 0; i < k; i++)
		{
			x[i] = nd(rng);
			y[i] = nd(rng);
			if (kind == 1) x[i] *= std::pow(10.0, -8.0 * (double)i / (double)k);
			if (kind == 2 && i % 2) { x[i] = -x[i - 1]; y[i] = y[i - 1] * (1 + 1e-10 * nd(rng)); }
			if (kind == 3) x[i] = 0;
			if (kind == 4) { x[i] = -value_of(0x3fefffffffffffffull); y[i] = value_of(0x3fe0808080808080ull); }
		}
		const double sx = std::ldexp(1.0, (int)(rng() % 200) - 100), sy = std::ldexp(1.0, (int)(rng() % 200) - 100);
		for (auto& v : x) v *= sx;
		for (auto& v : y) v *= sy;
		int E, F;
		const double r = slice_dot(x, y, E, F), ref = accurate_dot(x, y);
		const double tol = std::fabs(ref) * std::ldexp(1.0, -53) * 1.01 +
		                   (E && F ? (double)k * std::ldexp(1.0, E - 1022 + F - 1022 - 60) : 0.0);
		if (!(std::fabs(r - ref) <= tol)) bad++;
	}
	// tile lists
	for (int trial = 0; trial < 300; trial++)
	{
		auto rq = [&](i64 d, int w) { std::vector<q32> q((size_t)d); for (auto& x : q) x = (q32)(rng() % (2 * w + 1)) - w; return q; };
		const bool large = trial % 10 == 0;
		const int w = 1 + rng() % 2;
		const i64 da = 1 + rng() % (large ? 300 : 40), db = 1 + rng() % 5, dk = 1 + rng() % (large ? 900 : 60), dl = 1 + rng() % 4,
		          dc = 1 + rng() % (large ? 200 : 50);
		const std::vector<q32> qa = rq(da, w), qb = rq(db, 1), qk = rq(dk, w), ql = rq(dl, 1), qc = rq(dc, w);
		const int axs = rng() & 1, axt = rng() & 1;
		const int sk = (rng() & 1) ? 1 : -1, sl = (rng() & 1) ? 1 : -1;
		const i64 ds0[4] = {dk, dl, da, db}, ds1[4] = {da, db, dk, dl}, dt0[3] = {dk, dl, dc}, dt1[3] = {dc, dk, dl};
		const int rs0[4] = {sk, sl, 1, -1}, rs1[4] = {1, -1, sk, sl}, rt0[3] = {-sk, -sl, 1}, rt1[3] = {1, -sk, -sl};
		const Meta s = axs == AX_LEADING ? make_meta(4, ds0, rs0, {qk, ql, qa, qb}) : make_meta(4, ds1, rs1, {qa, qb, qk, ql});
		const Meta t = axt == AX_LEADING ? make_meta(3, dt0, rt0, {qk, ql, qc}) : make_meta(3, dt1, rt1, {qc, qk, ql});
		const int sms = trial % 3 == 0 ? 152 : 4;
		const DotLowering l = lower_dot(s, axs, t, axt, 2, GEMM_FP64, sms, nullptr, 64, true);
		const DotLowering f = lower_dot(s, axs, t, axt, 2, GEMM_FP64, sms);
		if (!l.tiles.empty() || !f.stiles.empty() || (f.tiles.empty() != l.stiles.empty())) bad++;
		if (l.cons.size() != f.cons.size() || l.outs.size() != f.outs.size()) bad++;
		// per output block: stages covered at every entry; its groups hold the terms of its contributions, in
		// their order
		std::vector<std::vector<i64>> cover(l.outs.size());
		std::vector<i64> stages(l.outs.size(), 0);
		for (size_t b = 0; b < l.outs.size(); b++)
		{
			const GemmOut& o = l.outs[b];
			cover[b].assign((size_t)o.m * o.n, 0);
			i64 k = 0;
			for (int c = o.c0; c < o.c0 + o.nc; c++) k += l.cons[(size_t)c].k;
			stages[b] = (k + SLICE_STAGE_K - 1) / SLICE_STAGE_K;
			if (o.nc == 0) continue;
			const SliceOut& so = l.souts[b];
			const int x = l.orient ? 0 : 1;
			for (int q = 0; q < 2; q++)
			{
				const SlicePack& sp = l.spack[q];
				const SliceGroup& g = sp.groups[(size_t)(q == x ? so.xgroup : so.ygroup)];
				const bool rows8 = q == x;
				if (g.rows != (q ? o.n : o.m) || g.ktot != k || g.nrun != o.nc) { bad++; continue; }
				if (g.base != (rows8 ? so.xbase : so.ybase)) bad++;
				if ((rows8 ? so.x8 : so.y32) != (rows8 ? (g.rows + 7) / 8 : (g.rows + 31) / 32)) bad++;
				const i64 bytes = stages[b] * (rows8 ? (i64)so.x8 * SLICE_ROW8_BYTES : (i64)so.y32 * SLICE_COL32_BYTES);
				if (g.base % 256 || g.base + bytes > sp.bytes) bad++;
				for (int c = 0; c < o.nc; c++)
				{
					const SliceRun& r = sp.runs[(size_t)(g.run0 + c)];
					const GemmContrib& n = l.cons[(size_t)(o.c0 + c)];
					if (r.k != n.k || r.off != (q ? n.b_off : n.a_off)) bad++;
					if ((g.rows > 1 && r.sr != (q ? n.sBn : n.sAm)) || (r.k > 1 && r.sk != (q ? n.sBk : n.sAk))) bad++;
				}
			}
		}
		// items: every 32 rows of a group by every SLICE_ITEM of its stages once, at the right term
		for (const SlicePack& sp : l.spack)
		{
			size_t at = 0;
			for (size_t gi = 0; gi < sp.groups.size(); gi++)
			{
				const SliceGroup& g = sp.groups[gi];
				for (int u0 = 0; u0 * SLICE_STAGE_K < g.ktot; u0 += SLICE_ITEM)
					for (int r0 = 0; r0 < g.rows; r0 += 32, at++)
					{
						if (at >= sp.items.size()) { bad++; continue; }
						const SliceItem& im = sp.items[at];
						int term = im.kk;
						for (int c = 0; c < im.run; c++) term += sp.runs[(size_t)(g.run0 + c)].k;
						if (im.group != (int)gi || im.row0 != r0 || im.u0 != u0 || term != u0 * SLICE_STAGE_K) bad++;
						if (im.run >= g.nrun || im.kk >= sp.runs[(size_t)(g.run0 + im.run)].k) bad++;
					}
			}
			if (at != sp.items.size()) bad++;
		}
		std::vector<int> shares(l.splits.size(), 0);
		int prev = 1 << 30;
		for (const SliceTile& T : l.stiles)
		{
			if ((T.u1 - T.u0) * T.halves > prev) bad++;
			prev = (T.u1 - T.u0) * T.halves;
			const GemmOut& o = l.outs[(size_t)T.out];
			const int rows = std::min(l.orient ? SLICE_TILE_ROWS : SLICE_TILE_COLS, o.m - T.m0);
			const int cols = std::min(l.orient ? SLICE_TILE_COLS : SLICE_TILE_ROWS, o.n - T.n0);
			if (rows < 1 || cols < 1) { bad++; continue; }
			if (T.halves != ((l.orient ? cols : rows) > SLICE_HALF ? 2 : 1)) bad++;
			if (T.u0 < 0 || T.u1 > stages[(size_t)T.out] || (o.nc > 0 && T.u0 >= T.u1)) bad++;
			if (o.nc > 0 && ((l.orient ? T.m0 : T.n0) / 8 >= l.souts[(size_t)T.out].x8 || (l.orient ? T.n0 : T.m0) / 32 >= l.souts[(size_t)T.out].y32)) bad++;
			if (T.split >= 0)
			{
				const GemmSplit& g = l.splits[(size_t)T.split];
				shares[(size_t)T.split]++;
				if (g.out != T.out || g.m0 != T.m0 || g.n0 != T.n0 || g.rows != rows || g.cols != cols || T.sp >= g.nsplit) bad++;
				if (g.part + (i64)g.nsplit * g.stride > l.work_doubles || 2 * ((g.rows - 1) * g.ld + g.cols) > g.stride) bad++;
			}
			for (int i = 0; i < rows; i++)
				for (int j = 0; j < cols; j++) cover[(size_t)T.out][(size_t)(T.m0 + i) * o.n + T.n0 + j] += std::max(T.u1 - T.u0, 1);
		}
		for (size_t b = 0; b < l.outs.size(); b++)
			for (i64 v : cover[b])
				if (v != std::max<i64>(stages[b], 1)) bad++;
		for (size_t q = 0; q < l.splits.size(); q++)
			if (shares[q] != l.splits[q].nsplit) bad++;
	}
	printf("mismatches: %d\n", bad);
	return bad != 0;
}
