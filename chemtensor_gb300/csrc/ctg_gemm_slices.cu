// ctg_gemm_slices.cu - FP64 block GEMM on the tensor cores by exact digit slices (ctg_slices.h).
//
// GB300 retires about two FP64 FMAs per clock and SM, its tensor cores about four thousand FP16 ones:
// the 36 digit products that stand for one FP64 product cost a fiftieth of the FMA. The sums over
// the digits are exact, so a result carries one rounding and the cut at 2^-62 of its two rows' largest
// entries (ctg_slices.h).
//
//   k_slice_exps   the largest exponent of every row of an operand (the scale of its digits)
//   k_slice_pack   cuts an operand into FP16 digits: per group of rows (the blocks with the same free
//                  indices) the terms of all its blocks one after the other, 16 terms at a time, in the
//                  canonical K-major core-matrix layout, so that a stage of the GEMM is two bulk copies.
//                  An entry is converted once here, and once per tile that reads it in the GEMM: with ten
//                  warps of the GEMM converting, its MMAs waited for them three quarters of the time
//   k_gemm_slices  persistent, one CTA per SM, output tiles of 128 x 64 (SliceTile): warp 0 copies the
//                  digits of 16 terms per stage (up to 32 + 16 KiB), warp 1 issues the MMAs, warps 4-19 add
//                  the orders up and write, and mark the results whose digits may not be enough
//   k_slice_find, k_slice_check, k_slice_parts   look at the marked results and sum those in FP64 that need it, one by
//                  one or, where a part of a tile has many, all of its results at a time; k_slice_lists makes lists of
//                  the nonzero terms of an MPO tensor or a small operand for them
// The 64 columns of a tile are two halves of 32 with an accumulator each in tensor memory: columns 32 o ..
// 32 o + 31 of it hold order o. Digit s of the 128 rows meets the digits 0 .. 7 - s of the 32 columns,
// which lie one after the other as rows of one B operand, in one MMA of N = 32 (8 - s) that writes
// the orders s .. 7: eight MMAs per half and 16 terms stand for 36 products, and the A digits are read
// once each. The tile is 64 wide because a stage then moves 48 KiB for 1240 cycles of MMAs (39 bytes a
// cycle and SM out of L2; 66 with 32 columns), and tensor memory holds no more. Every 128 terms the
// epilogue takes the sums over: half 0 while the MMAs of half 1 run, and conversely.
// Measured, three products of a local-Hamiltonian application at D = 1024 (4.1e9 FMAs): 7.65 ms on the
// FP64 pipe; 0.65 ms here (1.06 ms with the conversion inside the GEMM), 0.30 ms for the digits, 0.13 ms for the
// exponents and 0.25 ms for the marked results. The first two products are bound by the epilogue (integer
// instructions on 2e7 results, tensor pipe 28 and 37 % busy), the third, with ten times the terms, by the copies out
// of L2 (46 %). A molecular search (n = 16, D = 256): 1054 ms on the FP64 pipe, 214 ms here, 152 without the
// marked results.
// Every wait is bounded and ends when another warp has failed.
#include <algorithm>
#include <mutex>

#include "ctg_kernels.h"
#include "ctg_launch.cuh"
#include "ctg_slices.h"
#include "ctg_tcgen05.cuh"

namespace ctg {

namespace {

constexpr int SL_M = SLICE_TILE_ROWS, SL_HALF = SLICE_HALF;
constexpr int SL_EPI = 16, SL_EPI_WARP0 = 4;    // epilogue warps: a tensor-memory quarter by 8 columns of each half
constexpr int SL_THREADS = 32 * (SL_EPI_WARP0 + SL_EPI);
constexpr int SL_LBO = 128;                     // bytes between the two core matrices of 16 terms
constexpr int SL_A_SBO = SLICE_ROW8_BYTES, SL_B_SBO = 256;       // between groups of 8 rows
constexpr int SL_A_DIGIT = 256;                 // between the digits of a row
constexpr int SL_A_BYTES = SL_M / 8 * SLICE_ROW8_BYTES;          // 32 KiB
constexpr int SL_B_BYTES = 2 * SLICE_COL32_BYTES;                // 16 KiB
constexpr int SL_STAGE = SL_A_BYTES + SL_B_BYTES;
constexpr int SL_STAGES = 4;
constexpr int SL_ACC = SLICES * SL_HALF;        // accumulator columns of a half
constexpr int SL_FLUSH = SLICE_K / SLICE_STAGE_K;                // stages between flushes
constexpr int SL_LD = 5;                        // staging row of the epilogue (4 columns)
constexpr int SL_EPI_BYTES = SL_EPI * 32 * SL_LD * 8;
constexpr int SL_TILES = 32;                    // tiles described at a time (twice)
constexpr int SL_MASKS = SLICE_TILE_COLS * SL_M / 32;            // words of a tile's mask of suspect results
// one tile, as the other warps need it
struct SliceInfo {
	i64 xs, ys;                          // digits of its first stage (bytes)
	i64 co, sr0, sr1, sc0;               // output layout (GemmOut)
	int r1, c1;
	int tile;                            // -1: no more tiles
	int xstep, ystep, xbytes, ybytes;    // digits (bytes) between stages, and of one
	int nch, halves;
	int m0, n0, m, n;
	int split, sp;
	int xe, ye;                          // where the exponents of its rows begin
};
constexpr int SL_BARS = 2 * SL_STAGES + 4 + 4 + 1;
constexpr int SL_SMEM = SL_STAGES * SL_STAGE + SL_EPI_BYTES + 2 * SL_TILES * (int)sizeof(SliceInfo) + SL_BARS * 8 + 32;
constexpr int SL_WAIT = 1 << 21;                // polls before a wait is declared failed
// A description of 32 tiles lasts until the slowest warp has passed all of them; should one hang, its own wait
// ends first and sets the abort flag
constexpr int SL_INFO_WAITS = 2 * SL_TILES;
constexpr uint32_t SL_POLL_NS = 1000;           // longest a poll suspends its warp
static_assert(SL_SMEM <= 227 * 1024, "shared memory per CTA");
static_assert(2 * SL_ACC <= 512, "tensor memory");
static_assert((SL_EPI_WARP0 & 3) == 0, "a warp reads the tensor-memory quarter warp % 4");

// instruction descriptor: FP32 D, FP16 (format 0) K-major A and B, M = 128, N columns
__device__ __forceinline__ uint32_t slice_idesc(int n)
{
	return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(SL_M >> 4) << 24);
}

__device__ __forceinline__ bool elect_one()
{
	uint32_t p;
	asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(p));
	return p != 0;
}

__device__ __forceinline__ void slice_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate)
{
	asm volatile(
		"{\n\t.reg .pred p;\n\t"
		"setp.ne.b32 p, %4, 0;\n\t"
		"tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
		:
		: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate));
}

// bounded wait for the given phase parity; false after `limit` polls, or when *abort is set. Lanes may differ in
// what they see last: a warp that goes on together votes.
__device__ __forceinline__ bool slice_wait(uint64_t* bar, uint32_t parity, const volatile int* abort, int limit)
{
	const uint32_t mbar = smem_u32(bar);
	for (int it = 0; it < limit; it++)
	{
		uint32_t done;
		asm volatile(
			"{\n\t.reg .pred p;\n\t"
			"mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
			"selp.b32 %0, 1, 0, p;\n\t}"
			: "=r"(done)
			: "r"(mbar), "r"(parity), "r"(SL_POLL_NS)
			: "memory");
		if (done) return true;
		if (abort && *abort) return false;
	}
	return false;
}

// acc + x w for w = 2^24, 2^16, 2^8 or 1: one multiply-add instead of the shift and the two adds that a
// constant factor would become
__device__ __forceinline__ int64_t add_order(int64_t acc, int x, int w)
{
	int64_t r;
	asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(x), "r"(w), "l"(acc));
	return r;
}

// ------------------------------------------------------------------------------------
// exponents and digits of an operand
// ------------------------------------------------------------------------------------

// The items of an operand (32 rows of a group, a lane each, by SLICE_ITEM stages of its terms), 8 terms at a time.
struct SliceReader {
	const SliceRun* __restrict__ runs;   // the group's
	const double* x;
	const double* p;
	int row, nrun;
	bool valid;
	int c, kk, kend, sk;                 // place in the terms: block c of the group, term kk of it
	__device__ SliceReader(const SliceItem& im, const SliceGroup& g, const SliceRun* r, const double* entries, int row_)
		: runs(r + g.run0), x(entries), p(nullptr), row(row_), nrun(g.nrun), valid(row_ < g.rows), c(im.run - 1), kk(0), kend(0), sk(0)
	{
		next();
		kk = im.kk;
	}
	__device__ __forceinline__ void next()
	{
		kk = 0;
		if (++c < nrun)
		{
			const SliceRun r = runs[c];
			kend = r.k;
			sk = r.sk;
			p = x + r.off + (i64)(valid ? row : 0) * r.sr;
		}
	}
	// the next 8 terms, zeros past the end
	__device__ __forceinline__ void read8(double v[8])
	{
		if (c < nrun && kend - kk >= 8)
		{
			const double* s = p + (i64)kk * sk;
#pragma unroll
			for (int t = 0; t < 8; t++) v[t] = valid ? s[(i64)t * sk] : 0.0;
			kk += 8;
			if (kk == kend) next();
			return;
		}
#pragma unroll
		for (int t = 0; t < 8; t++)
		{
			v[t] = 0.0;
			if (c < nrun)
			{
				if (valid) v[t] = p[(i64)kk * sk];
				if (++kk == kend) next();
			}
		}
	}
};

constexpr int PACK_WARPS = 4;

// Largest exponent code of every row. A pass of its own: the rows' terms are spread over many items, and the
// digits need the whole row's code. It reads what the product before has just written, mostly from L2.
__global__ void __launch_bounds__(PACK_WARPS * 32)
k_slice_exps(int nitems, const SliceItem* __restrict__ items, const SliceGroup* __restrict__ groups,
             const SliceRun* __restrict__ runs, const double* x, int* codes, int* clear, int nclear)
{
	pdl_wait();
	pdl_trigger();
	for (int i = blockIdx.x * (PACK_WARPS * 32) + threadIdx.x; i < nclear; i += gridDim.x * (PACK_WARPS * 32)) clear[i] = 0;
	const int item = blockIdx.x * PACK_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
	if (item >= nitems) return;
	const SliceItem im = items[item];
	const SliceGroup g = groups[im.group];
	const int row = im.row0 + lane;
	SliceReader in(im, g, runs, x, row);
	const int n8 = 2 * min(SLICE_ITEM, (g.ktot + SLICE_STAGE_K - 1) / SLICE_STAGE_K - im.u0);
	uint32_t hi = 0, lo = 0;
	for (int u = 0; u < n8; u += 2)
	{
		double v[16];
		in.read8(v);
		in.read8(v + 8);
#pragma unroll
		for (int t = 0; t < 16; t++)
		{
			hi = max(hi, (uint32_t)__double2hiint(v[t]) & 0x7fffffffu);
			lo |= (uint32_t)__double2loint(v[t]);
		}
	}
	const int code = hi >= 0x00100000u ? (int)(hi >> 20) : (hi | lo) ? 1 : 0;
	if (code > 0) atomicMax(codes + g.row0 + row, code);
}

// bytes 0 and 1 (or 2 and 3) of w, biased digits u = d + 128 of two numbers, as FP16 pairs with the
// numbers' signs: 0x6400 + u is the FP16 pattern of 1024 + u, and sgn (1024 + u) - sgn 1152 = sgn d
__device__ __forceinline__ uint32_t digits_f16x2(uint32_t w, bool upper, uint32_t sgn, uint32_t off)
{
	const uint32_t p = __byte_perm(w, 0x64646464u, upper ? 0x4342 : 0x4140);
	uint32_t r;
	asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(p), "r"(sgn), "r"(off));
	return r;
}

// One warp per item, each lane a row: its 8 entries become 16 bytes of each of the 8 digits. The entries of the
// next 8 terms are on their way while these are cut.
__global__ void __launch_bounds__(PACK_WARPS * 32, 8)
k_slice_pack(int nitems, const SliceItem* __restrict__ items, const SliceGroup* __restrict__ groups,
             const SliceRun* __restrict__ runs, int rows8, const double* x, const int* codes, unsigned char* dst, short* exps)
{
	pdl_wait();
	pdl_trigger();
	const int item = blockIdx.x * PACK_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
	if (item >= nitems) return;
	const SliceItem im = items[item];
	const SliceGroup g = groups[im.group];
	const int row = im.row0 + lane;
	const int code = codes[g.row0 + row];
	if (im.u0 == 0) exps[g.row0 + row] = (short)slice_exp(code);
	// rows with smaller exponents are summed in FP64, or hold zeros only
	const int E = max(code, SLICE_EXP_MIN);
	// destination of the lane's row in stage 0, first 8 terms, digit 0; bytes between digits and stages
	unsigned char* out = dst + g.base + (lane & 7) * 16;
	const int groups8 = (g.rows + 7) / 8, groups32 = (g.rows + 31) / 32;
	const int digit = rows8 ? SL_A_DIGIT : SLICE_COL32_BYTES / SLICES;
	const i64 stage = rows8 ? (i64)groups8 * SLICE_ROW8_BYTES : (i64)groups32 * SLICE_COL32_BYTES;
	out += rows8 ? (i64)(row >> 3) * SLICE_ROW8_BYTES : (i64)(row >> 5) * SLICE_COL32_BYTES + (lane >> 3) * SL_B_SBO;
	const bool store = rows8 ? (row >> 3) < groups8 : true;
	SliceReader in(im, g, runs, x, row);
	const int stages = (g.ktot + SLICE_STAGE_K - 1) / SLICE_STAGE_K;
	const int n8 = 2 * min(SLICE_ITEM, stages - im.u0);
	out += (i64)im.u0 * stage;
	double v[8];
	in.read8(v);
	for (int u = 0; u < n8; u++)
	{
		uint32_t dig[8][2], sgn[4], off[4];
#pragma unroll
		for (int q = 0; q < 4; q++)
		{
			const uint32_t ha = (uint32_t)__double2hiint(v[2 * q]), hb = (uint32_t)__double2hiint(v[2 * q + 1]);
			const uint64_t da = slice_digits(ha, (uint32_t)__double2loint(v[2 * q]), E);
			const uint64_t db = slice_digits(hb, (uint32_t)__double2loint(v[2 * q + 1]), E);
			dig[2 * q][0] = (uint32_t)(da >> 32);
			dig[2 * q][1] = (uint32_t)da;
			dig[2 * q + 1][0] = (uint32_t)(db >> 32);
			dig[2 * q + 1][1] = (uint32_t)db;
			// +-1 and -+1152 in FP16, by the numbers' signs
			const uint32_t s2 = __byte_perm(ha, hb, 0x7030) & 0x80008000u;
			sgn[q] = s2 | 0x3c003c00u;
			off[q] = s2 ^ 0xe480e480u;
		}
		if (u + 1 < n8) in.read8(v);
		unsigned char* d = out + (i64)(u >> 1) * stage + (u & 1) * SL_LBO;
#pragma unroll
		for (int h = 0; h < 4; h++)
		{
			// digits 2 h and 2 h + 1: bytes 3 and 2 (h even) or 1 and 0 of word h / 2
			uint32_t w0[4], w1[4];
#pragma unroll
			for (int q = 0; q < 4; q++)
			{
				const uint32_t b = __byte_perm(dig[2 * q][h >> 1], dig[2 * q + 1][h >> 1], (h & 1) ? 0x4051 : 0x6273);
				w0[q] = digits_f16x2(b, false, sgn[q], off[q]);
				w1[q] = digits_f16x2(b, true, sgn[q], off[q]);
			}
			if (store)
			{
				*(uint4*)(d + 2 * h * digit) = make_uint4(w0[0], w0[1], w0[2], w0[3]);
				*(uint4*)(d + (2 * h + 1) * digit) = make_uint4(w1[0], w1[1], w1[2], w1[3]);
			}
		}
	}
}

// the nonzero terms of every row (a warp) of an item's 32
__global__ void __launch_bounds__(1024)
k_slice_lists(const SliceItem* __restrict__ items, const SliceGroup* __restrict__ groups, const SliceRun* __restrict__ runs,
              const double* x, SliceTerm* terms, int* counts)
{
	pdl_wait();
	pdl_trigger();
	const SliceItem im = items[blockIdx.x];
	if (im.u0 != 0) return;
	const SliceGroup g = groups[im.group];
	const int row = im.row0 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
	if (row >= g.rows) return;
	SliceTerm* list = terms + g.list + (i64)row * g.ktot;
	int n = 0;
	for (int c = 0; c < g.nrun; c++)
	{
		const SliceRun r = runs[g.run0 + c];
		const double* p = x + r.off + (i64)row * r.sr;
		for (int k0 = 0; k0 < r.k; k0 += 32)
		{
			const int k = k0 + lane;
			const double v = k < r.k ? p[(i64)k * r.sk] : 0.0;
			const unsigned some = __ballot_sync(0xffffffffu, v != 0.0);
			if (v != 0.0) list[n + __popc(some & ((1u << lane) - 1))] = SliceTerm{v, c, k};
			n += __popc(some);
		}
	}
	if (lane == 0) counts[g.row0 + row] = n;
}

// ------------------------------------------------------------------------------------
// the products
// ------------------------------------------------------------------------------------

__global__ void __launch_bounds__(SL_THREADS, 1)
k_gemm_slices(int ntiles, const SliceTile* tiles, const GemmOut* outs, const SliceOut* souts, const GemmContrib* cons,
              const GemmSplit* splits, int* counters, int orient, const double* A, const double* B, const unsigned char* xpack,
              const unsigned char* ypack, const short* xexps, const short* yexps, double* C, uint2* list, unsigned* masks, double* work, int* error, int limit)
{
	extern __shared__ __align__(1024) unsigned char smem[];
	double* stage_out = (double*)(smem + SL_STAGES * SL_STAGE);
	SliceInfo* infos = (SliceInfo*)((unsigned char*)stage_out + SL_EPI_BYTES);
	uint64_t* full = (uint64_t*)(infos + 2 * SL_TILES);                       // copies landed
	uint64_t* empty = full + SL_STAGES;                                       // MMAs of a stage done
	uint64_t* acc_full = empty + SL_STAGES;                                   // accumulators ready
	uint64_t* acc_empty = acc_full + 2;                                       // accumulators read
	uint64_t* info_full = acc_empty + 2;                                      // tiles described
	uint64_t* info_empty = info_full + 2;                                     // their descriptions read
	uint64_t* split_bar = info_empty + 2;                                     // epilogue: steps of a split tile
	uint32_t* tmem_slot = (uint32_t*)(split_bar + 1);
	volatile int* abort = (volatile int*)(tmem_slot + 1);
	volatile int* last_share = abort + 1;
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

	if (warp == 1)
	{
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512)
		             : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	if (tid == 0)
	{
		for (int st = 0; st < SL_STAGES; st++)
		{
			mbar_init(smem_u32(full + st), 1);
			mbar_init(smem_u32(empty + st), 1);
		}
		for (int b = 0; b < 2; b++)
		{
			mbar_init(smem_u32(acc_full + b), 1);
			mbar_init(smem_u32(acc_empty + b), SL_EPI);
			mbar_init(smem_u32(info_full + b), 1);
			mbar_init(smem_u32(info_empty + b), SL_EPI + 2);
		}
		mbar_init(smem_u32(split_bar), SL_EPI);
		*abort = 0;
	}
	asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = *tmem_slot;
	// everything up to here overlaps the tail of the previous kernel in the stream
	pdl_wait();
	// the list of k_slice_find, empty
	if (blockIdx.x == 0 && tid == 0) list[0] = make_uint2(0, 0);

	// the description of the CTA's tile number it (every lane of a warp, in order): null at the end
	auto tile_info = [&](int it, bool& ok) -> const SliceInfo* {
		const int batch = (it / SL_TILES) & 1;
		if (it % SL_TILES == 0) ok = __all_sync(0xffffffffu, slice_wait(info_full + batch, (uint32_t)((it / (2 * SL_TILES)) & 1), abort, SL_INFO_WAITS * limit));
		const SliceInfo* f = infos + batch * SL_TILES + it % SL_TILES;
		return ok && f->tile >= 0 ? f : nullptr;
	};
	// after the last use of it
	auto tile_done = [&](int it) {
		if (it % SL_TILES != SL_TILES - 1) return;
		__syncwarp();
		if (lane == 0) mbar_arrive(smem_u32(info_empty + ((it / SL_TILES) & 1)));
	};

	if (warp == 0)
	{
		// copies: the stages of every tile in order
		int g = 0;
		bool ok = true;
		for (int it = 0; ok; it++)
		{
			const SliceInfo* f = tile_info(it, ok);
			if (!f) break;
			const uint32_t xb = f->xbytes, yb = f->ybytes;
			const int xstep = f->xstep, ystep = f->ystep, nch = f->nch;
			const unsigned char *xs = xpack + f->xs, *ys = ypack + f->ys;
			for (int u = 0; u < nch; u++, g++, xs += xstep, ys += ystep)
			{
				const int st = g % SL_STAGES;
				if (g >= SL_STAGES) ok = slice_wait(empty + st, (uint32_t)(((g / SL_STAGES) - 1) & 1), abort, limit);
				ok = __all_sync(0xffffffffu, ok);
				if (!ok) break;
				if (lane == 0)
				{
					const uint32_t sa = smem_u32(smem + st * SL_STAGE), bar = smem_u32(full + st);
					mbar_expect_tx(bar, xb + yb);
					bulk_copy(sa, xs, xb, bar);
					bulk_copy(sa + SL_A_BYTES, ys, yb, bar);
				}
				__syncwarp();
			}
			tile_done(it);
		}
		if (!ok && lane == 0)
		{
			*abort = 1;
			atomicExch(error, 1);
		}
		// the copies of the last stages must land before shared memory is released
		for (int u = max(g - SL_STAGES, 0); u < g; u++) slice_wait(full + u % SL_STAGES, (uint32_t)((u / SL_STAGES) & 1), nullptr, SL_WAIT);
	}
	else if (warp == 1)
	{
		// the whole warp walks the stages (its state stays in uniform registers), one lane issues
		int g = 0, f = 0;                  // stages, flushes of a half
		bool ok = true;
		const bool one = elect_one();
		const uint32_t s0 = smem_u32(smem);
		for (int it = 0; ok; it++)
		{
			const SliceInfo* info = tile_info(it, ok);
			if (!info) break;
			const int nch = info->nch, halves = info->halves;
			for (int u = 0; u < nch && ok; u++)
			{
				const int st = g % SL_STAGES;
				const bool first = u % SL_FLUSH == 0, last = u % SL_FLUSH == SL_FLUSH - 1 || u == nch - 1;
				ok = __all_sync(0xffffffffu, slice_wait(full + st, (uint32_t)((g / SL_STAGES) & 1), abort, limit));
				if (!ok) break;
				for (int h = 0; h < halves; h++)
				{
					const int fh = f + h, b = fh & 1;
					if (first && fh >= 2)
					{
						ok = __all_sync(0xffffffffu, slice_wait(acc_empty + b, (uint32_t)(((fh >> 1) - 1) & 1), abort, limit));
						if (!ok)
						{
							// what has been issued of the stage still ends in its commit
							if (h > 0 && one) mma_commit(smem_u32(empty + st));
							if (h > 0) g++;
							break;
						}
					}
					tc_fence_after();
					if (one)
					{
						const uint64_t da = make_desc(s0 + st * SL_STAGE, SL_LBO, SL_A_SBO);
						const uint64_t db = make_desc(s0 + st * SL_STAGE + SL_A_BYTES + h * SLICE_COL32_BYTES, SL_LBO, SL_B_SBO);
						const uint32_t acc = tmem + (uint32_t)(b * SL_ACC);
#pragma unroll
						for (int s = 0; s < SLICES; s++)
							slice_mma(acc + (uint32_t)(s * SL_HALF), da + (uint64_t)(s * (SL_A_DIGIT >> 4)), db,
							          slice_idesc(SL_HALF * (SLICES - s)), s > 0 || !first);
						if (last) mma_commit(smem_u32(acc_full + b));
						if (h == halves - 1) mma_commit(smem_u32(empty + st));
					}
					__syncwarp();
				}
				if (last) f += halves;
				if (ok) g++;
			}
			tile_done(it);
		}
		if (!ok && lane == 0)
		{
			*abort = 1;
			atomicExch(error, 1);
		}
		// no MMA may still run when tensor memory is freed
		if (g > 0) slice_wait(empty + (g - 1) % SL_STAGES, (uint32_t)(((g - 1) / SL_STAGES) & 1), nullptr, SL_WAIT);
		pdl_trigger();
	}
	else if (warp == 2)
	{
		// descriptions, 32 tiles at a time, one per lane: no other warp waits for global memory but for its
		// data. Tiles come in order of falling work; each pass over the CTAs reverses the order of the
		// one before
		const int grid = gridDim.x, me = blockIdx.x, npass = (ntiles + grid - 1) / grid;
		bool ok = true;
		for (int p0 = 0; ok; p0 += SL_TILES)
		{
			const int batch = (p0 / SL_TILES) & 1;
			if (p0 >= 2 * SL_TILES)
				ok = __all_sync(0xffffffffu, slice_wait(info_empty + batch, (uint32_t)((p0 / (2 * SL_TILES) - 1) & 1), abort, SL_INFO_WAITS * limit));
			if (!ok) break;
			const int pass = p0 + lane, ti = pass * grid + ((pass & 1) ? grid - 1 - me : me);
			SliceInfo f = {};
			f.tile = -1;
			if (pass < npass && ti < ntiles)
			{
				const SliceTile t = tiles[ti];
				const GemmOut o = outs[t.out];
				f.tile = ti;
				f.nch = t.u1 - t.u0;
				f.halves = t.halves;
				f.m0 = t.m0;
				f.n0 = t.n0;
				f.m = o.m;
				f.n = o.n;
				f.co = o.c_off;
				f.sr0 = o.sr0;
				f.sr1 = o.sr1;
				f.sc0 = o.sc0;
				f.r1 = o.r1;
				f.c1 = o.c1;
				f.split = t.split;
				f.sp = t.sp;
				if (f.nch > 0)
				{
					const SliceOut s = souts[t.out];
					const int x8 = (orient ? t.m0 : t.n0) >> 3, y32 = (orient ? t.n0 : t.m0) >> 5;
					f.xstep = s.x8 * SLICE_ROW8_BYTES;
					f.ystep = s.y32 * SLICE_COL32_BYTES;
					f.xbytes = min(SL_M / 8, s.x8 - x8) * SLICE_ROW8_BYTES;
					f.ybytes = min(2, s.y32 - y32) * SLICE_COL32_BYTES;
					f.xs = s.xbase + (i64)t.u0 * f.xstep + (i64)x8 * SLICE_ROW8_BYTES;
					f.ys = s.ybase + (i64)t.u0 * f.ystep + (i64)y32 * SLICE_COL32_BYTES;
					f.xe = s.xrow + x8 * 8;
					f.ye = s.yrow + y32 * 32;
				}
			}
			infos[batch * SL_TILES + lane] = f;
			__syncwarp();
			if (lane == 0) mbar_arrive(smem_u32(info_full + batch));
			if (p0 + SL_TILES > npass) break;      // the batch had a lane without a tile: the end is marked
		}
		if (!ok && lane == 0)
		{
			*abort = 1;
			atomicExch(error, 1);
		}
	}
	else if (warp >= SL_EPI_WARP0)
	{
		const int q = warp & 3, part = (warp - SL_EPI_WARP0) >> 2;
		const int gr = q * 32 + lane;                          // MMA row
		double* sw = stage_out + (warp - SL_EPI_WARP0) * 32 * SL_LD;
		int f = 0, nsp = 0;
		int wt[4] = {1 << 24, 1 << 16, 1 << 8, 1};
		asm("" : "+r"(wt[0]), "+r"(wt[1]), "+r"(wt[2]), "+r"(wt[3]));
		// the sums of the halves between the flushes of a tile with several
		int64_t kept[32];
		bool ok = true;
		for (int it = 0; ok; it++)
		{
			const SliceInfo* info = tile_info(it, ok);
			if (!info) break;
			const SliceInfo& tile = *info;
			const int nch = tile.nch, halves = tile.halves;
			// MMA rows of this warp inside the output block
			const int rows = min(32, (orient ? tile.m - tile.m0 : tile.n - tile.n0) - q * 32);
			const int nfl = max((nch + SL_FLUSH - 1) / SL_FLUSH, 1);
			// a last flush of 32 terms at most (32 x 7 x 2^14 < 2^22) leaves the integers in the low bits of
			// sum + 1.5 2^23: minus the offsets that their patterns will add, 0x4b400000 times the weights
			// (the sums of the orders 0 .. 2 stay below 2^22 for 128 terms, and always go that way: the integer
			// conversion runs at an eighth of the rate)
			const bool few_last = nch > 0 && (nch - 1) % SL_FLUSH < 2;
			// (modulo 2^64, as the sums: the offsets pass 63 bits at 437 flushes, the orders themselves do not before
			// SLICE_TERMS_MAX terms)
			const int64_t start_hi = (int64_t)(0ull - 0x4b400000ull * ((uint64_t)nfl * 0x01010100ull + (few_last ? 1 : 0)));
			const int64_t start_lo = few_last ? -0x4b400000ll * 0x01010101ll : 0;
			for (int fl = 0; fl < nfl && ok; fl++)
			{
#pragma unroll 1
				for (int h = 0; h < halves; h++)
				{
					// MMA columns of this warp; one without columns waits and arrives like the others, so that no
					// warp gets more than a phase of a barrier ahead or behind
					const int gc = h * SL_HALF + part * 8;
					const int cols = min(8, (orient ? tile.n - tile.n0 : tile.m - tile.m0) - gc);
					const bool active = rows > 0 && cols > 0;
					int64_t hi[8], lo[8];
					if (fl == 0)
					{
#pragma unroll
						for (int c = 0; c < 8; c++)
						{
							hi[c] = start_hi;
							lo[c] = start_lo;
						}
					}
					else
					{
#pragma unroll
						for (int c = 0; c < 8; c++)
						{
							hi[c] = kept[h * 16 + c];
							lo[c] = kept[h * 16 + 8 + c];
						}
					}
					// exponents of the lane's row and of the 8 columns, for the results
					int e = 0;
					int4 ys = make_int4(0, 0, 0, 0);
					if (fl == nfl - 1 && tile.split < 0 && nch > 0 && active)
					{
						if (lane < rows) e = xexps[tile.xe + gr];
						ys = *(const int4*)(yexps + tile.ye + gc);
					}
					if (nch > 0)
					{
						const int b = f & 1;
						ok = __all_sync(0xffffffffu, slice_wait(acc_full + b, (uint32_t)((f >> 1) & 1), abort, limit));
						f++;
						if (!ok) break;
						if (active)
						{
							tc_fence_after();
							const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * SL_ACC + part * 8);
							const bool few = few_last && fl == nfl - 1;
#pragma unroll
							for (int op = 0; op < SLICES; op += 2)
							{
								uint32_t v[16];
								asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
								             : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
								             : "r"(ta + (uint32_t)(op * SL_HALF)));
								asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
								             : "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
								             : "r"(ta + (uint32_t)((op + 1) * SL_HALF)));
								asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
								for (int c = 0; c < 16; c++)
								{
									const float x = __uint_as_float(v[c]);
									v[c] = few || op + c / 8 <= 2 ? __float_as_uint(x + 12582912.0f) : (uint32_t)__float2int_rn(x);
								}
								// orders op and op + 1 have the weights 2^24, 2^16 (op % 4 == 0) or 2^8, 1 in their half
								const int w0 = (op & 2) ? wt[2] : wt[0], w1 = (op & 2) ? wt[3] : wt[1];
#pragma unroll
								for (int c = 0; c < 8; c++)
								{
									int64_t& acc = op < 4 ? hi[c] : lo[c];
									acc = add_order(add_order(acc, (int)v[c], w0), (int)v[8 + c], w1);
								}
							}
							tc_fence_before();
						}
						__syncwarp();
						if (lane == 0) mbar_arrive(smem_u32(acc_empty + b));
					}
					if (fl < nfl - 1)
					{
#pragma unroll
						for (int c = 0; c < 8; c++)
						{
							kept[h * 16 + c] = hi[c];
							kept[h * 16 + 8 + c] = lo[c];
						}
						continue;
					}
					if (!active) continue;
					if (tile.split >= 0)
					{
						// a share of a split tile: its sums as they are
						const GemmSplit sp = splits[tile.split];
						int64_t* w = (int64_t*)(work + sp.part + (i64)tile.sp * sp.stride);
						if (lane < rows)
						{
#pragma unroll
							for (int c = 0; c < 8; c++)
								if (c < cols) *(longlong2*)(w + 2 * ((gc + c) * SL_M + gr)) = make_longlong2(hi[c], lo[c]);
						}
						continue;
					}
					// results in place of the sums, and which of them k_slice_check has to look at
					unsigned mask = 0;
#pragma unroll
					for (int c = 0; c < 8; c++)
					{
						const int w = c < 2 ? ys.x : c < 4 ? ys.y : c < 6 ? ys.z : ys.w;
						const int fc = (c & 1) ? w >> 16 : (int)(short)w;
						hi[c] = nch > 0 ? (int64_t)slice_value(hi[c], lo[c], slice_top(e, fc)) : 0;
						const unsigned m = __ballot_sync(0xffffffffu, lane < rows && slice_suspect(e, fc, (int)(hi[c] >> 52) & 0x7ff));
						if (lane == c) mask = m;
					}
					if (lane < 8) masks[(i64)tile.tile * SL_MASKS + (gc + lane) * 4 + q] = mask;
					if (orient == 0)
					{
						// lanes are neighbouring columns of the output block: coalesced
						if (lane < rows)
						{
							const int j = tile.n0 + gr, jq = j / tile.c1, r1 = tile.r1;
							const i64 sr1 = tile.sr1, wrap = tile.sr0 - (i64)(r1 - 1) * sr1;
							const int i = tile.m0 + gc, ih = i / r1;
							int il = i - ih * r1;
							double* ci = C + tile.co + (i64)jq * tile.sc0 + (j - jq * tile.c1) + (i64)ih * tile.sr0 + (i64)il * sr1;
#pragma unroll
							for (int c = 0; c < 8; c++)
							{
								if (c < cols) *ci = __longlong_as_double(hi[c]);
								// the next row: a step inside the run of low row indices, or past its end
								const bool end = ++il == r1;
								ci += end ? wrap : sr1;
								if (end) il = 0;
							}
						}
					}
					else
					{
						// lanes are rows of the output block: turned in shared memory, so that 4 lanes write 4
						// neighbouring columns of a row
						const int i = min(tile.m0 + gr, tile.m - 1), iq = i / tile.r1;
						const i64 ro = tile.co + (i64)iq * tile.sr0 + (i64)(i - iq * tile.r1) * tile.sr1;
						const int c = lane & 3;
#pragma unroll
						for (int c0 = 0; c0 < 8; c0 += 4)
						{
							if (cols <= c0) break;
#pragma unroll
							for (int t = 0; t < 4; t++) sw[lane * SL_LD + t] = __longlong_as_double(hi[c0 + t]);
							__syncwarp();
							const int j = tile.n0 + gc + min(c0 + c, cols - 1), jq = j / tile.c1;
							const i64 co = (i64)jq * tile.sc0 + (j - jq * tile.c1);
#pragma unroll
							for (int t = 0; t < 4; t++)
							{
								const int rr = t * 8 + (lane >> 2);
								const i64 rof = __shfl_sync(0xffffffffu, ro, rr);
								if (rr < rows && c0 + c < cols) C[rof + co] = sw[rr * SL_LD + c];
							}
							__syncwarp();
						}
					}
					__syncwarp();
				}
			}
			if (!ok) break;
			if (tile.split >= 0)
			{
				// the CTA that completes a split tile last adds the shares (integers of one scale) and rounds
				const GemmSplit sp = splits[tile.split];
				auto step = [&]() {
					__syncwarp();
					if (lane == 0) mbar_arrive(smem_u32(split_bar));
					ok = __all_sync(0xffffffffu, slice_wait(split_bar, (uint32_t)(nsp & 1), abort, limit));
					nsp++;
				};
				__threadfence();
				step();
				if (!ok) break;
				if (warp == SL_EPI_WARP0 && lane == 0) *last_share = atomicAdd(counters + tile.split, 1) == sp.nsplit - 1;
				step();
				if (!ok) break;
				if (*last_share)
				{
					__threadfence();
					// a warp per column and 32 rows of the MMA tile
					const GemmOut o = outs[sp.out];
					const int mr = orient ? sp.rows : sp.cols, mc = orient ? sp.cols : sp.rows;
					unsigned* mask = masks + (i64)(ntiles + tile.split) * SL_MASKS;
					for (int wd = warp - SL_EPI_WARP0; wd < 4 * mc; wd += SL_EPI)
					{
						const int col = wd >> 2, row = (wd & 3) * 32 + lane;
						if ((wd & 3) * 32 >= mr) continue;
						bool look = false;
						if (row < mr)
						{
							const longlong2* pw = (const longlong2*)(work + sp.part) + col * SL_M + row;
							int64_t hi = 0, lo = 0;
							for (int p = 0; p < sp.nsplit; p++)
							{
								const longlong2 v = __ldcg(pw + (i64)p * (sp.stride / 2));
								hi += v.x;
								lo += v.y;
							}
							const int e = xexps[tile.xe + row], fc = yexps[tile.ye + col];
							const uint64_t r = slice_value(hi, lo, slice_top(e, fc));
							look = slice_suspect(e, fc, (int)(r >> 52) & 0x7ff);
							C[gemm_out_index(o, sp.m0 + (orient ? row : col), sp.n0 + (orient ? col : row))] = __longlong_as_double((long long)r);
						}
						const unsigned m = __ballot_sync(0xffffffffu, look);
						if (lane == 0) mask[wd] = m;
					}
					if (tid == 32 * SL_EPI_WARP0) counters[tile.split] = 0;
				}
				// nobody overwrites *last_share before every warp has read it
				step();
				if (!ok) break;
			}
			tile_done(it);
		}
		if (!ok && lane == 0)
		{
			*abort = 1;
			atomicExch(error, 1);
		}
	}
	tc_fence_before();
	__syncthreads();
	if (warp == 1)
	{
		tc_fence_after();
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
	}
}

// ------------------------------------------------------------------------------------
// the results whose digits may not be enough
// ------------------------------------------------------------------------------------

// Results of rows that are not finite, tiny or out of range are FP64 sums over the operands. A small result keeps
// its value if one of its terms is large (terms that cancel); if none is (a graded row times a column that is small
// where the row is large), it is an FP64 sum too, so that every entry has the accuracy of the FP64 pipe.
// k_slice_find lists the mask words with suspects, so that the few tiles that hold many are shared out;
// k_slice_check takes the words in turn, a warp each, its lanes divided among the word's suspects.
// Suspect: 0.6 % of random operands (all of them cleared by their first terms), 5 % in a molecular search at
// D = 256, of which 3 % are summed: there the MPO tensor's rows have ten nonzero terms of four hundred, and the lists
// of these (k_slice_lists) stand for the row.
constexpr int CHECK_WARPS = 4, CHECK_UNROLL = 4;
// rows per listed word, 32 or fewer where the sums are long (max_k is the longest one of the product)
__host__ __device__ inline int check_rows(int k) { return k >= 2048 ? 1 : k >= 512 ? 8 : 32; }

__device__ __forceinline__ int biased_exponent(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// rows and columns of the MMA tile of a mask (numbers below ntiles: tiles that are not split; then split tiles)
struct MaskTile {
	int out, m0, n0, mr, mc;
	__device__ MaskTile(int id, int ntiles, const SliceTile* tiles, const GemmSplit* splits, const GemmOut* outs, int orient)
	{
		mr = mc = 0;
		if (id < ntiles)
		{
			const SliceTile t = tiles[id];
			if (t.split >= 0 || t.u0 == t.u1) return;
			out = t.out;
			m0 = t.m0;
			n0 = t.n0;
		}
		else
		{
			const GemmSplit t = splits[id - ntiles];
			out = t.out;
			m0 = t.m0;
			n0 = t.n0;
		}
		const int m = outs[out].m - m0, n = outs[out].n - n0;
		mr = min(SL_M, orient ? m : n);
		mc = min(SLICE_TILE_COLS, orient ? n : m);
	}
};

// A part of a tile, 32 MMA rows by 8 columns, of which many results are suspect, such as those of a row that is
// graded against the other operand's columns, is summed as a whole, its operands read once for all of it
// (k_slice_parts). The words keep the parts if these are too few to fill the SMs (two for each). A result of the words
// costs 4 to 6 times the terms that one of a part costs, 1.3 to 2.7 times with lists. Products of which all results are
// suspect (ms by words, by parts, on the FP64 pipe): 2048 x 2048 x 2048 terms 90, 14.0, 14.3; with lists
// 512 x 4096 x 2048 20.4, 7.0, 7.5; 4096 x 512 x 2048 9.4, 7.0, 7.5. From half the results on, with lists or without,
// the molecular search (n = 24, D = 512) is slower by 2 %: there the words of long sums read the same terms at a time.
constexpr double CHECK_WHOLE = 3, CHECK_WHOLE_LISTS = 1.25;
constexpr int CHECK_TERMS = 32, PARTS_SM = 5;

// list: the numbers of its words and parts (zero before the launch), then (mask word, its bits); from its end, the
// parts (of mask word by column group, rows: 32 id + 4 group + rows)
__global__ void __launch_bounds__(CHECK_WARPS * 32)
k_slice_find(int ntiles, int nsplits, const SliceTile* __restrict__ tiles, const GemmOut* __restrict__ outs,
             const SliceOut* __restrict__ souts, const GemmSplit* __restrict__ splits, int orient, int swap,
             const SliceGroup* __restrict__ groups, const int* counts, const unsigned* masks, uint2* list, unsigned last)
{
	pdl_wait();
	pdl_trigger();
	const int lane = threadIdx.x & 31, units = (ntiles + nsplits) * 8;
	for (int unit = blockIdx.x * CHECK_WARPS + (threadIdx.x >> 5); unit < units; unit += gridDim.x * CHECK_WARPS)
	{
		const int id = unit >> 3, col = (unit & 7) * 8 + (lane >> 2), row0 = (lane & 3) * 32;
		const MaskTile t(id, ntiles, tiles, splits, outs, orient);
		const unsigned at = (unsigned)id * SL_MASKS + (unit & 7) * 32 + lane;
		unsigned word = col < t.mc && row0 < t.mr ? masks[at] : 0;
		if (t.mr - row0 < 32) word &= (1u << max(t.mr - row0, 0)) - 1;
		if (!__any_sync(0xffffffffu, word != 0)) continue;
		const SliceOut so = souts[t.out];
		// the suspects of the lane's 32 rows, and their terms: with lists, as many as a row of them has here
		auto sum = [](int v) {
			for (int q = 4; q < 32; q <<= 1) v += __shfl_xor_sync(0xffffffffu, v, q);
			return v;
		};
		const int cols = min(8, t.mc - (unit & 7) * 8), nrow = min(32, t.mr - row0);
		const double suspects = (counts ? CHECK_WHOLE_LISTS : CHECK_WHOLE) * sum(__popc(word)), whole = 32.0 * cols * so.k;
		bool part = suspects * so.k > whole;
		if (counts && __any_sync(0xffffffffu, part))
		{
			const bool rows = swap != orient;
			const int* len = counts + groups[rows ? so.xgroup : so.ygroup].row0 + (rows == (orient != 0) ? t.m0 : t.n0) + (rows ? row0 : (unit & 7) * 8);
			const int nlen = rows ? nrow : cols;
			int n = 0;
			for (int r = lane >> 2; r < nlen; r += 8) n += len[r];
			const double terms = sum(n);
			part = part && suspects * terms > whole * nlen;
		}
		if (part)
		{
			if (lane < 4) list[last - atomicAdd(&list[0].y, 1u)] = make_uint2((unsigned)unit * 4 + lane, 0);
			word = 0;
		}
		const int width = check_rows(so.k);
		int n = 0;
		for (int q = 0; q < 32; q += width) n += (word >> q & (0xffffffffu >> (32 - width))) != 0;
		int end = n;
#pragma unroll
		for (int q = 1; q < 32; q <<= 1)
		{
			const int v = __shfl_up_sync(0xffffffffu, end, q);
			if (lane >= q) end += v;
		}
		unsigned base = 0;
		if (lane == 31) base = atomicAdd(&list[0].x, (unsigned)end);
		base = __shfl_sync(0xffffffffu, base, 31) + 1 + end - n;
		for (int q = 0; q < 32; q += width)
		{
			const unsigned part = word & (0xffffffffu >> (32 - width)) << q;
			if (part) list[base++] = make_uint2(at, part);
		}
	}
}

// use(a, b) for the terms of an entry that are the lane's (sub, sub + lanes, ..), for all lanes of a warp at once,
// until done() holds in all of them. x is the MPO tensor, whose rows are mostly zeros, or else the operand with fewer
// entries (i its row), and read first: unless all terms are asked for, y is read where x is not zero, and terms that
// are zero in every lane are left out. Contributions of more terms than an entry has lanes are taken one by one;
// those of shorter ones, 32 at a time, are one list.
template <bool ALL, class Use, class Done>
__device__ __forceinline__ void entry_terms(const GemmOut& o, const GemmContrib* cons, bool swap, const double* x, const double* y, int i,
                                            int j, int sub, int lanes, bool on, const Use& use, const Done& done)
{
	constexpr unsigned FULL = 0xffffffffu;
	const int lane = threadIdx.x & 31;
	for (int c0 = 0; c0 < o.nc; c0 += 32)
	{
		const int nb = min(32, o.nc - c0);
		GemmContrib g = {};
		if (lane < nb) g = cons[o.c0 + c0 + lane];
		if (swap) g = GemmContrib{g.b_off, g.a_off, g.k, g.sBn, g.sBk, g.sAk, g.sAm};
		int end = g.k;
#pragma unroll
		for (int q = 1; q < 32; q <<= 1)
		{
			const int v = __shfl_up_sync(FULL, end, q);
			if (lane >= q) end += v;
		}
		const int start = end - g.k, total = __shfl_sync(FULL, end, 31);
		const bool list = total < nb * lanes;
		for (int c = 0; c < (list ? 1 : nb); c++)
		{
			const int n = list ? total : __shfl_sync(FULL, g.k, c);
			int d = c;
			auto first = [&] { return x + __shfl_sync(FULL, g.a_off, d) + (i64)i * __shfl_sync(FULL, g.sAm, d); };
			auto second = [&] { return y + __shfl_sync(FULL, g.b_off, d) + (i64)j * __shfl_sync(FULL, g.sBn, d); };
			const double *px = first(), *py = second();
			int kx = __shfl_sync(FULL, g.sAk, d), ky = __shfl_sync(FULL, g.sBk, d);
			for (int t0 = 0; t0 < n; t0 += CHECK_UNROLL * lanes)
			{
				double a[CHECK_UNROLL], b[CHECK_UNROLL];
				const double* pb[CHECK_UNROLL];
#pragma unroll
				for (int u = 0; u < CHECK_UNROLL; u++)
				{
					int t = t0 + u * lanes + sub;
					const bool in = on && t < n;
					if (list)
					{
						d = 0;
#pragma unroll
						for (int step = 16; step > 0; step >>= 1)
							if (__shfl_sync(FULL, start, d + step) <= t) d += step;
						px = first();
						py = second();
						kx = __shfl_sync(FULL, g.sAk, d);
						ky = __shfl_sync(FULL, g.sBk, d);
						t -= __shfl_sync(FULL, start, d);
					}
					pb[u] = in ? py + (i64)t * ky : nullptr;
					a[u] = in ? px[(i64)t * kx] : 0.0;
				}
#pragma unroll
				for (int u = 0; u < CHECK_UNROLL; u++) b[u] = pb[u] && (ALL || a[u] != 0.0) ? *pb[u] : 0.0;
#pragma unroll
				for (int u = 0; u < CHECK_UNROLL; u++)
					if (ALL || __any_sync(FULL, a[u] != 0.0)) use(a[u], b[u]);
				if (done()) return;
			}
		}
	}
}

// The parts of k_slice_find, a block each: 32 terms at a time, a quarter of them for each warp, a lane's row by 8 columns.
// Bound by the FP64 pipe (a warp's FMA takes 64 clocks of a quarter of the SM, beside a row's entry and 8 staged ones).
__global__ void __launch_bounds__(CHECK_WARPS * 32, PARTS_SM)
k_slice_parts(int ntiles, const SliceTile* __restrict__ tiles, const GemmOut* __restrict__ outs, const SliceOut* __restrict__ souts,
              const GemmContrib* __restrict__ cons, const GemmSplit* __restrict__ splits, int orient, const double* A, const double* B,
              const short* xexps, const short* yexps, const unsigned* masks, double* C, const uint2* list, unsigned last, unsigned least)
{
	__shared__ double stage[CHECK_TERMS][8], sums[CHECK_WARPS - 1][8][32];
	__shared__ unsigned cleared[32];
	pdl_wait();
	pdl_trigger();
	const unsigned nparts = list[0].y;
	if (nparts < least) return;
	for (unsigned p = blockIdx.x; p < nparts; p += gridDim.x)
	{
		const unsigned part = list[last - p].x;
		const int id = (int)(part >> 5), c0 = (int)(part >> 2 & 7) * 8, q0 = (int)(part & 3);
		const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = q0 * 32 + lane;
		const MaskTile t(id, ntiles, tiles, splits, outs, orient);
		const GemmOut o = outs[t.out];
		const SliceOut so = souts[t.out];
		const int cols = min(8, t.mc - c0), xr = (orient ? t.m0 : t.n0) + row, yr = (orient ? t.n0 : t.m0) + c0;
		const bool in = row < t.mr;
		const int e = in ? xexps[so.xrow + xr] : 0;
		unsigned left = 0, look = 0;           // results that are suspect and not cleared; those in range
		int limit[8], most[8];
		double s[8];
	#pragma unroll
		for (int c = 0; c < 8; c++)
		{
			s[c] = 0.0;
			limit[c] = most[c] = 0;
			if (!in || c >= cols || !(masks[(unsigned)id * SL_MASKS + (c0 + c) * 4 + q0] >> lane & 1)) continue;
			const int f = yexps[so.yrow + yr + c];
			limit[c] = slice_term_limit(e, f);
			left |= 1u << c;
			look |= (unsigned)slice_in_range(slice_top(e, f)) << c;
		}
		if (warp == 0) cleared[lane] = 0;
		// a sum that may overflow stays one chain (see k_slice_check): the first warp's
		const bool chain = __syncthreads_or((left & ~look) != 0);
		const int u0 = chain ? 0 : warp * (CHECK_TERMS / CHECK_WARPS), u1 = chain ? (warp ? 0 : CHECK_TERMS) : u0 + CHECK_TERMS / CHECK_WARPS;
		const int st = threadIdx.x & (CHECK_TERMS - 1), sc = (threadIdx.x / CHECK_TERMS) * 2;
		bool some = true;
		for (int q = 0; q < o.nc && some; q++)
		{
			const GemmContrib g = cons[o.c0 + q];
			const double* px = orient ? A + g.a_off + (i64)xr * g.sAm : B + g.b_off + (i64)xr * g.sBn;
			const double* py = orient ? B + g.b_off + (i64)yr * g.sBn : A + g.a_off + (i64)yr * g.sAm;
			const int kx = orient ? g.sAk : g.sBk, ky = orient ? g.sBk : g.sAk, ny = orient ? g.sBn : g.sAm;
			for (int k0 = 0; k0 < g.k; k0 += CHECK_TERMS)
			{
				const int n = min(CHECK_TERMS, g.k - k0);
				// the warps have read the stage before; a result that one of them has cleared is done
				some = __syncthreads_or(left != 0);
				if (!some) break;
				left &= ~cleared[lane];
	#pragma unroll
				for (int c = 0; c < 2; c++)
					stage[st][sc + c] = st < n && sc + c < cols ? py[(i64)(k0 + st) * ky + (i64)(sc + c) * ny] : 0.0;
				__syncthreads();
				for (int u = u0; u < min(n, u1); u += CHECK_UNROLL)
				{
					double x[CHECK_UNROLL];
	#pragma unroll
					for (int v = 0; v < CHECK_UNROLL; v++) x[v] = in && u + v < n ? px[(i64)(k0 + u + v) * kx] : 0.0;
	#pragma unroll
					for (int v = 0; v < CHECK_UNROLL; v++)
					{
						if (u + v >= n) break;
						const int ex = biased_exponent(x[v]);
	#pragma unroll
						for (int c = 0; c < 8; c++)
						{
							const double y = stage[u + v][c];
							s[c] = fma(x[v], y, s[c]);
							most[c] = max(most[c], ex + biased_exponent(y));
						}
					}
				}
				unsigned enough = 0;
	#pragma unroll
				for (int c = 0; c < 8; c++) enough |= (unsigned)(most[c] >= limit[c]) << c;
				enough &= left & look;
				if (enough) atomicOr(&cleared[lane], enough);
				left &= ~enough;
			}
		}
		if (warp > 0)
		{
	#pragma unroll
			for (int c = 0; c < 8; c++) sums[warp - 1][c][lane] = s[c];
		}
		__syncthreads();
		if (warp == 0)
		{
			left &= ~cleared[lane];
	#pragma unroll
			for (int c = 0; c < 8; c++)
			{
				double r = s[c];
				if (!chain)
					for (int w = 0; w < CHECK_WARPS - 1; w++) r += sums[w][c][lane];
				if (left >> c & 1) C[orient ? gemm_out_index(o, xr, yr + c) : gemm_out_index(o, yr + c, xr)] = r;
			}
		}
		__syncthreads();
	}
}

__global__ void __launch_bounds__(CHECK_WARPS * 32)
k_slice_check(int ntiles, const SliceTile* __restrict__ tiles, const GemmOut* __restrict__ outs, const SliceOut* __restrict__ souts,
              const GemmContrib* __restrict__ cons, const GemmSplit* __restrict__ splits, int orient, int swap,
              const SliceGroup* __restrict__ groups, const SliceTerm* terms, const int* counts, const double* A, const double* B,
              const short* xexps, const short* yexps, const unsigned* masks, double* C, const uint2* list, unsigned last, unsigned least, unsigned pieces)
{
	pdl_wait();
	pdl_trigger();
	const int lane = threadIdx.x & 31;
	const unsigned nword = list[0].x, nparts = list[0].y;
	const unsigned n = nword + (nparts < least ? nparts * 8 * pieces : 0);
	// an entry of the list, or a piece of a part's word
	auto word_at = [&](unsigned at) -> uint2 {
		if (at < nword) return list[1 + at];
		const unsigned v = at - nword, p = list[last - v / (8 * pieces)].x, col = (p >> 2 & 7) * 8 + v / pieces % 8, row0 = (p & 3) * 32;
		const MaskTile t((int)(p >> 5), ntiles, tiles, splits, outs, orient);
		if ((int)col >= t.mc) return make_uint2(0, 0);
		const unsigned wd = (p >> 5) * SL_MASKS + col * 4 + (p & 3);
		const int rows = min(32, t.mr - (int)row0);
		return make_uint2(wd, masks[wd] & 0xffffffffu >> (32 - rows) & 0xffffffffu >> (32 - 32 / pieces) << (v % pieces * (32 / pieces)));
	};
	// the operand that is read first, and the other one
	const double *x = swap ? B : A, *y = swap ? A : B;
	unsigned item = blockIdx.x * CHECK_WARPS + (threadIdx.x >> 5);
	uint2 next = item < n ? word_at(item) : make_uint2(0, 0);
	for (; item < n; item += gridDim.x * CHECK_WARPS)
	{
		const uint2 w = next;
		if (item + gridDim.x * CHECK_WARPS < n) next = word_at(item + gridDim.x * CHECK_WARPS);
		if (w.y == 0) continue;
		const int wd = (int)(w.x % SL_MASKS), col = wd >> 2;
		const MaskTile t((int)(w.x / SL_MASKS), ntiles, tiles, splits, outs, orient);
		const GemmOut o = outs[t.out];
		const SliceOut so = souts[t.out];
		// the suspects get 32, 16, .. 1 lanes each
		const int count = __popc(w.y), lanes = 32 >> (count > 1 ? 32 - __clz(count - 1) : 0);
		const int which = lane / lanes, sub = lane % lanes;
		unsigned left = w.y;
		for (int q = 0; q < which && q + 1 < count; q++) left &= left - 1;
		const int row = (wd & 3) * 32 + __ffs(left) - 1;
		const int i = orient ? t.m0 + row : t.m0 + col, j = orient ? t.n0 + col : t.n0 + row;
		const int ix = swap ? j : i, iy = swap ? i : j;
		const int e = xexps[so.xrow + (orient ? i : j)], f = yexps[so.yrow + (orient ? j : i)], limit = slice_term_limit(e, f);
		const unsigned mine = (lanes == 32 ? 0xffffffffu : (1u << lanes) - 1) << (which * lanes);
		const bool on = which < count, look = on && slice_in_range(slice_top(e, f));
		bool enough = false;
		double s = 0.0;
		if (terms)
		{
			// test and sum in one
			const SliceGroup g = groups[swap == orient ? so.ygroup : so.xgroup];
			const SliceTerm* p = terms + g.list + (i64)ix * g.ktot;
			const int k = look ? counts[g.row0 + ix] : 0;
			for (int t0 = sub; __any_sync(0xffffffffu, t0 < k && !enough); t0 += CHECK_UNROLL * lanes)
			{
				SliceTerm z[CHECK_UNROLL];
				double v[CHECK_UNROLL];
#pragma unroll
				for (int u = 0; u < CHECK_UNROLL; u++) z[u] = t0 + u * lanes < k ? p[t0 + u * lanes] : SliceTerm{0.0, 0, 0};
#pragma unroll
				for (int u = 0; u < CHECK_UNROLL; u++)
				{
					v[u] = 0.0;
					if (t0 + u * lanes >= k) continue;
					const GemmContrib h = cons[o.c0 + z[u].run];
					v[u] = swap ? y[h.a_off + (i64)iy * h.sAm + (i64)z[u].k * h.sAk] : y[h.b_off + (i64)iy * h.sBn + (i64)z[u].k * h.sBk];
				}
#pragma unroll
				for (int u = 0; u < CHECK_UNROLL; u++)
				{
					enough |= biased_exponent(z[u].v) + biased_exponent(v[u]) >= limit;
					s = fma(z[u].v, v[u], s);
				}
				enough = (__ballot_sync(0xffffffffu, enough && look) & mine) != 0;
			}
		}
		else if (__any_sync(0xffffffffu, look))
			entry_terms<false>(o, cons, swap, x, y, ix, iy, sub, lanes, look,
			                   [&](double a, double b) { enough |= biased_exponent(a) + biased_exponent(b) >= limit; },
			                   [&] {
				                   enough = (__ballot_sync(0xffffffffu, enough && look) & mine) != 0;
				                   return !__any_sync(0xffffffffu, look && !enough);
			                   });
		const auto all = [] { return false; };
		const bool sum = look && !enough;
		if (__any_sync(0xffffffffu, sum))
		{
			if (!terms)
				entry_terms<false>(o, cons, swap, x, y, ix, iy, sub, lanes, sum, [&](double a, double b) { s = fma(a, b, s); }, all);
			for (int q = lanes >> 1; q > 0; q >>= 1) s += __shfl_xor_sync(0xffffffffu, s, q);
		}
		// a sum that may overflow in one chain: infinities of both signs would make NaN of partial sums
		const bool chain = on && !look && sub == 0;
		if (__any_sync(0xffffffffu, chain))
		{
			if (chain) s = 0.0;
			entry_terms<true>(o, cons, swap, x, y, ix, iy, 0, 1, chain, [&](double a, double b) { if (chain) s = fma(a, b, s); }, all);
		}
		if ((sum && sub == 0) || chain) C[gemm_out_index(o, i, j)] = s;
	}
}

}  // namespace

// the list, then the masks
i64 slice_check_bytes(int ntiles, int nsplits, int max_k)
{
	return 8 + (i64)(ntiles + nsplits) * SL_MASKS * (32 / check_rows(max_k) * (i64)sizeof(uint2) + (i64)sizeof(unsigned));
}

// last entry of the list
static i64 check_last(int ntiles, int nsplits, int max_k) { return (i64)(ntiles + nsplits) * SL_MASKS * (32 / check_rows(max_k)); }
static unsigned* check_masks(void* check, int ntiles, int nsplits, int max_k)
{
	return (unsigned*)((uint2*)check + 1 + check_last(ntiles, nsplits, max_k));
}

void launch_slice_exps(int nitems, const SliceItem* items, const SliceGroup* groups, const SliceRun* runs, const double* x,
                       int* codes, int* clear, int nclear, cudaStream_t st)
{
	if (nitems <= 0) return;
	launch_pdl(launch_config(dim3((nitems + PACK_WARPS - 1) / PACK_WARPS), dim3(PACK_WARPS * 32), 0, st), k_slice_exps, nitems, items,
	           groups, runs, x, codes, clear, nclear);
}

void launch_slice_pack(int nitems, const SliceItem* items, const SliceGroup* groups, const SliceRun* runs, bool rows8,
                       const double* x, const int* codes, void* dst, short* exps, cudaStream_t st)
{
	if (nitems <= 0) return;
	launch_pdl(launch_config(dim3((nitems + PACK_WARPS - 1) / PACK_WARPS), dim3(PACK_WARPS * 32), 0, st), k_slice_pack, nitems, items,
	           groups, runs, rows8 ? 1 : 0, x, codes, (unsigned char*)dst, exps);
}

void launch_slice_lists(int nitems, const SliceItem* items, const SliceGroup* groups, const SliceRun* runs, const double* x,
                        SliceTerm* terms, int* counts, cudaStream_t st)
{
	if (nitems > 0) launch_pdl(launch_config(dim3(nitems), dim3(1024), 0, st), k_slice_lists, items, groups, runs, x, terms, counts);
}

void launch_gemm_slices(int ntiles, const SliceTile* tiles, const GemmOut* outs, const SliceOut* souts, const GemmContrib* cons,
                        int nsplits, const GemmSplit* splits, int* counters, int orient, const double* A, const double* B,
                        const void* xpack, const void* ypack, const short* xexps, const short* yexps, double* C, int max_k,
                        void* check, double* work, int* error, int num_sms, cudaStream_t st)
{
	if (ntiles <= 0) return;
	// the attribute belongs to the device
	static std::once_flag attr_once[64];
	int dev = 0;
	CTG_CUDA(cudaGetDevice(&dev));
	std::call_once(attr_once[dev & 63], [] {
		CTG_CUDA(cudaFuncSetAttribute(k_gemm_slices, cudaFuncAttributeMaxDynamicSharedMemorySize, SL_SMEM));
	});
	// persistent: one CTA per SM (its shared memory admits one)
	const cudaLaunchConfig_t cfg = launch_config(dim3(std::min(ntiles, num_sms)), dim3(SL_THREADS), SL_SMEM, st);
	launch_pdl(cfg, k_gemm_slices, ntiles, tiles, outs, souts, cons, splits, counters, orient, A, B, (const unsigned char*)xpack,
	           (const unsigned char*)ypack, xexps, yexps, C, (uint2*)check, check_masks(check, ntiles, nsplits, max_k), work, error,
	           (int)std::min<long long>(tc_wait_limit(), SL_WAIT));
}

void launch_slice_check(int ntiles, int nsplits, const SliceTile* tiles, const GemmOut* outs, const SliceOut* souts,
                        const GemmContrib* cons, const GemmSplit* splits, int orient, bool b_smaller, const SliceGroup* groups,
                        const SliceTerm* terms, const int* counts, const double* A, const double* B, const short* xexps,
                        const short* yexps, double* C, int max_k, void* check, int num_sms, cudaStream_t st)
{
	if (ntiles <= 0) return;
	uint2* list = (uint2*)check;
	const int all = num_sms * 8;
	const unsigned* masks = check_masks(check, ntiles, nsplits, max_k);
	const unsigned last = (unsigned)check_last(ntiles, nsplits, max_k);
	launch_pdl(launch_config(dim3(std::min((ntiles + nsplits) * 8 / CHECK_WARPS, 2 * all)), dim3(CHECK_WARPS * 32), 0, st), k_slice_find,
	           ntiles, nsplits, tiles, outs, souts, splits, orient, b_smaller ? 1 : 0, groups, terms ? counts : nullptr, masks, list, last);
	launch_pdl(launch_config(dim3(all), dim3(CHECK_WARPS * 32), 0, st), k_slice_check, ntiles, tiles, outs, souts, cons, splits, orient,
	           b_smaller ? 1 : 0, groups, terms, counts, A, B, xexps, yexps, masks, C, list, last,
	           2u * num_sms, (unsigned)(32 / check_rows(max_k)));
	launch_pdl(launch_config(dim3(num_sms * PARTS_SM), dim3(CHECK_WARPS * 32), 0, st), k_slice_parts, ntiles, tiles, outs, souts, cons, splits,
	           orient, A, B, xexps, yexps, masks, C, list, last, 2u * num_sms);
}

}  // namespace ctg
