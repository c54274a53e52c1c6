// ctg_kernels.cu - FP64 grouped block GEMM and the block data-movement kernels.
#include "ctg_kernels.h"
#include "ctg_launch.cuh"

namespace ctg {

// ------------------------------------------------------------------------------------
// grouped FP64 block GEMM (plain path; dense_tensor_dot_update, dense_tensor.c:1761-1837)
// ------------------------------------------------------------------------------------

constexpr int GEMM_THREADS = 256;     // 16 x 16 thread grid for every tile class
constexpr int GEMM_BK = 16;           // terms per stage
constexpr int GEMM_TERMS = 64;        // terms whose operand positions are tabulated at a time
constexpr int GEMM_RING = 2 * GEMM_BK * (128 + 1 + 8 + 1);      // entries of the ring of stages, real product
constexpr int GEMM_RING_Z = GEMM_BK * (128 + 1 + 8 + 1);        // complex entries

// The sum of a tile runs over its contributions and each one's inner index. GEMM_TERMS consecutive terms of
// that one list are tabulated: where the term's column of A and row of B lie.
struct GemmTerms {
	i64 a[GEMM_TERMS], b[GEMM_TERMS];
	int sa[GEMM_TERMS], sb[GEMM_TERMS];
	int start[GEMM_TERMS];            // first term of the contributions, scratch of the tabulation
	GemmContrib con[GEMM_TERMS];
	int half;                         // terms of the first 32 contributions
	int count, next_c, next_k;        // terms tabulated; where the list goes on
	int a_by_k, b_by_k;               // consecutive terms are consecutive entries
};

// The next (at most GEMM_TERMS) terms from contribution c, inner index k on. All threads call it; the first
// 64 take a contribution each, add up the terms before theirs and look up their own term's contribution.
__device__ __forceinline__ void gemm_terms(GemmTerms& w, const GemmTile& tile, const GemmContrib* __restrict__ cons, int c, int k)
{
	const int tid = threadIdx.x, lane = tid & 31;
	if (c == tile.c1)
	{
		// the last (mostly the only) contribution: its terms follow one another, nothing to add up or look up
		const GemmContrib g = cons[c];
		if (tid < GEMM_TERMS)
		{
			w.a[tid] = g.a_off + (i64)(k + tid) * g.sAk;
			w.b[tid] = g.b_off + (i64)(k + tid) * g.sBk;
			w.sa[tid] = g.sAm;
			w.sb[tid] = g.sBn;
		}
		if (tid == 0)
		{
			const bool whole = tile.k1 - k <= GEMM_TERMS;
			w.count = whole ? tile.k1 - k : GEMM_TERMS;
			w.next_c = whole ? c + 1 : c;
			w.next_k = k + GEMM_TERMS;
			w.a_by_k = g.sAk == 1 && g.sAm != 1;
			w.b_by_k = g.sBk == 1 && g.sBn != 1;
		}
		__syncthreads();
		return;
	}
	int n = 0, incl = 0;
	if (tid < GEMM_TERMS)
	{
		if (c + tid <= tile.c1)
		{
			const GemmContrib g = cons[c + tid];
			w.con[tid] = g;
			n = (c + tid == tile.c1 ? tile.k1 : g.k) - (tid == 0 ? k : 0);
		}
		incl = n;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1)
		{
			const int v = __shfl_up_sync(0xffffffffu, incl, o);
			if (lane >= o) incl += v;
		}
		if (tid == 31) w.half = incl;
	}
	__syncthreads();
	if (tid < GEMM_TERMS)
	{
		if (tid >= 32) incl += w.half;
		const int first = incl - n;
		w.start[tid] = first;
		// the contribution with the table's last term, or the last one of all
		if (n > 0 && first < GEMM_TERMS && (incl >= GEMM_TERMS || c + tid == tile.c1))
		{
			const bool whole = incl <= GEMM_TERMS;
			w.count = whole ? incl : GEMM_TERMS;
			w.next_c = whole ? c + tid + 1 : c + tid;
			w.next_k = whole ? 0 : GEMM_TERMS - first + (tid == 0 ? k : 0);
		}
		if (tid == 0)
		{
			if (c > tile.c1) w.count = 0;
			w.a_by_k = n > 0 && w.con[0].sAk == 1 && w.con[0].sAm != 1;
			w.b_by_k = n > 0 && w.con[0].sBk == 1 && w.con[0].sBn != 1;
		}
	}
	__syncthreads();
	if (tid < w.count)
	{
		int j = 0;
#pragma unroll
		for (int step = GEMM_TERMS / 2; step > 0; step >>= 1)
			if (w.start[j + step] <= tid) j += step;
		const GemmContrib g = w.con[j];
		const int kk = tid - w.start[j] + (j == 0 ? k : 0);
		w.a[tid] = g.a_off + (i64)kk * g.sAk;
		w.b[tid] = g.b_off + (i64)kk * g.sBk;
		w.sa[tid] = g.sAm;
		w.sb[tid] = g.sBn;
	}
	__syncthreads();
}

__device__ __forceinline__ void gemm_copy(double* dst, const double* src)
{
	asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void gemm_copy(double2* dst, const double2* src)
{
	asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void gemm_copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void gemm_copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// entry arithmetic of the tiles: T = double, or double2 for complex128. `flip` has the sign bit set
// where the operand is conjugated.
__device__ __forceinline__ double gemm_entry(double x, unsigned) { return x; }
__device__ __forceinline__ double2 gemm_entry(double2 x, unsigned flip)
{
	return make_double2(x.x, __hiloint2double(__double2hiint(x.y) ^ (int)flip, __double2loint(x.y)));
}
// A complex sum is kept as the sums of Re a times b and of Im a times b, so that a pair of entries takes four FMAs
// and the sum no more rounding than with products that are rounded by themselves; where the accumulators of a tile
// would not fit (SMALL = false), those take six instructions.
struct GemmPair {
	double2 p, q;
};
template <class T, bool SMALL> struct GemmAcc { using type = T; };
template <> struct GemmAcc<double2, true> { using type = GemmPair; };
__device__ __forceinline__ void gemm_mac(double& c, double a, double b) { c = fma(a, b, c); }
__device__ __forceinline__ void gemm_mac(double2& c, double2 a, double2 b)
{
	c.x += fma(a.x, b.x, -(a.y * b.y));
	c.y += fma(a.x, b.y, a.y * b.x);
}
__device__ __forceinline__ void gemm_mac(GemmPair& c, double2 a, double2 b)
{
	c.p.x = fma(a.x, b.x, c.p.x);
	c.p.y = fma(a.x, b.y, c.p.y);
	c.q.x = fma(a.y, b.x, c.q.x);
	c.q.y = fma(a.y, b.y, c.q.y);
}
__device__ __forceinline__ double gemm_value(double c) { return c; }
__device__ __forceinline__ double2 gemm_value(double2 c) { return c; }
__device__ __forceinline__ double2 gemm_value(const GemmPair& c) { return make_double2(c.p.x - c.q.y, c.p.y + c.q.x); }
__device__ __forceinline__ void gemm_add(double& c, double x) { c += x; }
__device__ __forceinline__ void gemm_add(double2& c, double2 x)
{
	c.x += x.x;
	c.y += x.y;
}

template <class T, int RING, int BM, int BN, int TM, int TN>
__device__ __forceinline__ void gemm_tile(const GemmTile& tile, const GemmOut* __restrict__ outs,
                                          const GemmContrib* __restrict__ cons, const GemmSplit* __restrict__ splits,
                                          int* __restrict__ counters, const T* __restrict__ A, const T* __restrict__ B,
                                          T* __restrict__ C, T* __restrict__ work, T* sm, GemmTerms& w, unsigned fa, unsigned fb)
{
	constexpr int NTX = BN / TN, NTY = BM / TM, NT = NTX * NTY, BK = GEMM_BK;
	constexpr int STAGE = BK * (BM + 1 + BN + 1);
	constexpr int NST = RING / STAGE < GEMM_TERMS / BK ? RING / STAGE : GEMM_TERMS / BK;      // stages in flight
	static_assert(NT == GEMM_THREADS && NST >= 1, "tile class layout");
	const GemmOut o = outs[tile.out];
	const int tid = threadIdx.x;
	const int tx = tid % NTX, ty = tid / NTX;
	using Acc = typename GemmAcc<T, TM * TN <= 4>::type;
	Acc acc[TM][TN];
#pragma unroll
	for (int i = 0; i < TM; i++)
#pragma unroll
		for (int j = 0; j < TN; j++) acc[i][j] = Acc();

	// rows and columns beyond the block and terms beyond the table stay unset: what they give is not stored
	auto load = [&](int st) {
		T* as = sm + (st % NST) * STAGE;
		T* bs = as + BK * (BM + 1);
		const int k0 = st * BK;
#pragma unroll
		for (int e = tid; e < BM * BK; e += NT)
		{
			const int kk = w.a_by_k ? e % BK : e / BM, i = w.a_by_k ? e / BK : e % BM;
			if (k0 + kk < w.count && tile.m0 + i < o.m)
				gemm_copy(as + kk * (BM + 1) + i, A + w.a[k0 + kk] + (i64)(tile.m0 + i) * w.sa[k0 + kk]);
		}
#pragma unroll
		for (int e = tid; e < BN * BK; e += NT)
		{
			const int kk = w.b_by_k ? e % BK : e / BN, j = w.b_by_k ? e / BK : e % BN;
			if (k0 + kk < w.count && tile.n0 + j < o.n)
				gemm_copy(bs + kk * (BN + 1) + j, B + w.b[k0 + kk] + (i64)(tile.n0 + j) * w.sb[k0 + kk]);
		}
	};
	bool first = true;
	for (int c = tile.c0, k = tile.k0; first || c <= tile.c1;)
	{
		gemm_terms(w, tile, cons, c, k);
		// the lists belong to the plan: the operands are the first access that has to wait for the kernel before
		if (first)
		{
			pdl_wait();
			pdl_trigger();
			first = false;
		}
		const int count = w.count, nst = (count + BK - 1) / BK;
		if (count == 0) break;
#pragma unroll
		for (int st = 0; st < NST; st++)
		{
			if (st < nst) load(st);
			gemm_copy_commit();
		}
		for (int st = 0; st < nst; st++)
		{
			gemm_copy_wait<NST - 1>();
			__syncthreads();
			const T* as = sm + (st % NST) * STAGE;
			const T* bs = as + BK * (BM + 1);
			const int kmax = min(BK, count - st * BK);
			for (int kk = 0; kk < kmax; kk++)
			{
				T av[TM], bv[TN];
#pragma unroll
				for (int i = 0; i < TM; i++) av[i] = gemm_entry(as[kk * (BM + 1) + ty + i * NTY], fa);
#pragma unroll
				for (int j = 0; j < TN; j++) bv[j] = gemm_entry(bs[kk * (BN + 1) + tx + j * NTX], fb);
#pragma unroll
				for (int i = 0; i < TM; i++)
#pragma unroll
					for (int j = 0; j < TN; j++) gemm_mac(acc[i][j], av[i], bv[j]);
			}
			if (st + NST < nst)
			{
				__syncthreads();
				load(st + NST);
			}
			gemm_copy_commit();
		}
		c = w.next_c;
		k = w.next_k;
		__syncthreads();                  // the table and the ring are free again
	}
	if (tile.split >= 0)
	{
		// partial sum of a split tile (full BM x BN, leading dimension BN); the CTA that completes
		// the split last adds the partial sums in a fixed order (deterministic) and writes C
		const GemmSplit sp = splits[tile.split];
		T* part = work + sp.part + (i64)tile.sp * sp.stride;
#pragma unroll
		for (int i = 0; i < TM; i++)
#pragma unroll
			for (int j = 0; j < TN; j++) part[(ty + i * NTY) * BN + tx + j * NTX] = gemm_value(acc[i][j]);
		__threadfence();
		__syncthreads();
		__shared__ int last;
		if (tid == 0) last = atomicAdd(counters + tile.split, 1) == sp.nsplit - 1;
		__syncthreads();
		if (!last) return;
		__threadfence();
		for (int e = tid; e < sp.rows * sp.cols; e += NT)
		{
			const int i = e / sp.cols, j = e - i * sp.cols;
			const T* pw = work + sp.part + (i64)i * sp.ld + j;
			// in four runs (a fraction of the rounding of one chain) or in one
			const int run = sp.chain ? sp.nsplit : (sp.nsplit + 3) / 4;
			T sum = T();
#pragma unroll 1
			for (int q0 = 0; q0 < sp.nsplit; q0 += run)
			{
				T part_sum = T();
#pragma unroll 4
				for (int q = q0; q < min(q0 + run, sp.nsplit); q++) gemm_add(part_sum, __ldcg(pw + (i64)q * sp.stride));
				gemm_add(sum, part_sum);
			}
			C[gemm_out_index(o, sp.m0 + i, sp.n0 + j)] = sum;
		}
		if (tid == 0) counters[tile.split] = 0;
		return;
	}
#pragma unroll
	for (int i = 0; i < TM; i++)
	{
		const int gi = tile.m0 + ty + i * NTY;
		if (gi >= o.m) continue;
#pragma unroll
		for (int j = 0; j < TN; j++)
		{
			const int gj = tile.n0 + tx + j * NTX;
			if (gj < o.n) C[gemm_out_index(o, gi, gj)] = gemm_value(acc[i][j]);
		}
	}
}

template <class T, int RING, bool LARGE>
__device__ __forceinline__ void gemm_any_tile(const GemmTile& tile, const GemmOut* __restrict__ outs,
                                              const GemmContrib* __restrict__ cons, const GemmSplit* __restrict__ splits,
                                              int* __restrict__ counters, const T* __restrict__ A, const T* __restrict__ B,
                                              T* __restrict__ C, T* __restrict__ work, unsigned fa, unsigned fb)
{
	__shared__ T sm[RING];
	__shared__ GemmTerms w;
	if (LARGE && tile.cls == TILE_L)
	{
		gemm_tile<T, RING, 64, 64, 4, 4>(tile, outs, cons, splits, counters, A, B, C, work, sm, w, fa, fb);
		return;
	}
	switch (tile.cls)
	{
	case TILE_M: gemm_tile<T, RING, 32, 32, 2, 2>(tile, outs, cons, splits, counters, A, B, C, work, sm, w, fa, fb); break;
	case TILE_W: gemm_tile<T, RING, 16, 64, 1, 4>(tile, outs, cons, splits, counters, A, B, C, work, sm, w, fa, fb); break;
	case TILE_T: gemm_tile<T, RING, 64, 16, 4, 1>(tile, outs, cons, splits, counters, A, B, C, work, sm, w, fa, fb); break;
	case TILE_R8: gemm_tile<T, RING, 8, 32, 1, 1>(tile, outs, cons, splits, counters, A, B, C, work, sm, w, fa, fb); break;
	case TILE_R4: gemm_tile<T, RING, 4, 64, 1, 1>(tile, outs, cons, splits, counters, A, B, C, work, sm, w, fa, fb); break;
	case TILE_C8: gemm_tile<T, RING, 32, 8, 1, 1>(tile, outs, cons, splits, counters, A, B, C, work, sm, w, fa, fb); break;
	case TILE_C4: gemm_tile<T, RING, 64, 4, 1, 1>(tile, outs, cons, splits, counters, A, B, C, work, sm, w, fa, fb); break;
	case TILE_W8: gemm_tile<T, RING, 8, 128, 1, 4>(tile, outs, cons, splits, counters, A, B, C, work, sm, w, fa, fb); break;
	case TILE_T8: gemm_tile<T, RING, 128, 8, 4, 1>(tile, outs, cons, splits, counters, A, B, C, work, sm, w, fa, fb); break;
	default: gemm_tile<T, RING, 16, 16, 1, 1>(tile, outs, cons, splits, counters, A, B, C, work, sm, w, fa, fb); break;
	}
}

// Bound by the FP64 pipe where the blocks are large, by latency where they are small: a tile's chain is tile,
// contributions, operands, FMAs, result, and only the last two use the pipe. So
//   - the lists are read before the wait on the kernel before (they belong to the plan);
//   - up to 64 terms are one flat list over all contributions, staged by asynchronous copies with up to four
//     stages in flight: short contributions (k of 1 to 20) share stages and latency. Staging each
//     contribution by itself, every load exposed, took as long per contribution as now per tile;
//   - tiles come longest first and split shares are small (see lower_dot): the SMs' FP64 times of one product
//     had differed by 29 to 81 percent of its duration.
// Clock stamps in a product of 891 tiles of one to thirteen terms: 2100 cycles to the table, 1050 to the
// operands, 3500 of FMAs (five blocks on the SM), 700 to the result. Four blocks per SM for LARGE = false:
// 94.0 ms of a spin-chain search and 69.8 of a Hubbard one (D = 100) against 95.4 and 71.4 with five, 94.8
// and 72.8 with six and a ring of half the size.
// Before and after, all of it: Hubbard L = 32, D = 256 search 286 -> 269 ms, D = 100 74.0 -> 69.8, spin chain
// L = 20, D = 32 98.5 -> 94.0, one-site Hubbard D = 256 69.3 -> 68.1.
// LARGE: the product has TILE_L tiles.
template <bool LARGE>
__global__ void __launch_bounds__(GEMM_THREADS, LARGE ? 3 : 4)
k_gemm_f64(const GemmTile* __restrict__ tiles, const GemmOut* __restrict__ outs, const GemmContrib* __restrict__ cons,
           const GemmSplit* __restrict__ splits, int* __restrict__ counters, const double* __restrict__ A,
           const double* __restrict__ B, double* __restrict__ C, double* __restrict__ work)
{
	gemm_any_tile<double, GEMM_RING, LARGE>(tiles[blockIdx.x], outs, cons, splits, counters, A, B, C, work, 0u, 0u);
}

// complex128: the tiles, split shares and lists of the real product, four FMAs per pair of entries.
// Bound by the FP64 pipe on large blocks and by latency on small ones (tens of blocks of 1 to 60 rows).
// A tile of its own, 32 x 32 with all contributions on one CTA, left most SMs idle and spent six FP64
// instructions per pair: 164 us per product of a Hubbard chain at bond dimension 64 (628 products,
// 103 ms), 20 us with the work lists' narrow tiles and split shares (12.7 ms). Two blocks per SM: the
// 4 x 4 complex accumulators and operands of TILE_L need 128 registers.
__global__ void __launch_bounds__(GEMM_THREADS, 2)
k_gemm_z(const GemmTile* __restrict__ tiles, const GemmOut* __restrict__ outs, const GemmContrib* __restrict__ cons,
         const GemmSplit* __restrict__ splits, int* __restrict__ counters, const double2* __restrict__ A,
         const double2* __restrict__ B, double2* __restrict__ C, double2* __restrict__ work, unsigned flip_a, unsigned flip_b)
{
	gemm_any_tile<double2, GEMM_RING_Z, true>(tiles[blockIdx.x], outs, cons, splits, counters, A, B, C, work, flip_a, flip_b);
}

int tile_rows(int cls)
{
	return TILE_ROWS[cls];
}

int tile_cols(int cls)
{
	return TILE_COLS[cls];
}

void launch_gemm_f64(int ntiles, const GemmTile* tiles, const GemmOut* outs, const GemmContrib* cons,
                     const GemmSplit* splits, int* counters, const double* A, const double* B, double* C, double* work,
                     cudaStream_t st, double flops, bool large)
{
	if (ntiles <= 0) return;
	// programmatic dependent launch for the short products of a sweep (tens of microseconds); a
	// product of milliseconds gains nothing from it and lost 2 % with it (the next kernel's blocks
	// scheduled beside its last waves)
	const cudaLaunchConfig_t cfg = launch_config(dim3(ntiles), dim3(GEMM_THREADS), 0, st);
	const auto kernel = large ? k_gemm_f64<true> : k_gemm_f64<false>;
	if (flops < 2e8) launch_pdl(cfg, kernel, tiles, outs, cons, splits, counters, A, B, C, work);
	else CTG_CUDA(cudaLaunchKernelEx(&cfg, kernel, tiles, outs, cons, splits, counters, A, B, C, work));
}

void launch_gemm_z(int ntiles, const GemmTile* tiles, const GemmOut* outs, const GemmContrib* cons,
                   const GemmSplit* splits, int* counters, const double* A, const double* B, double* C, double* work,
                   bool conj_a, bool conj_b, cudaStream_t st, double flops)
{
	if (ntiles <= 0) return;
	const cudaLaunchConfig_t cfg = launch_config(dim3(ntiles), dim3(GEMM_THREADS), 0, st);
	const double2 *a = (const double2*)A, *b = (const double2*)B;
	double2 *o = (double2*)C, *w = (double2*)work;
	const unsigned fa = conj_a ? 0x80000000u : 0u, fb = conj_b ? 0x80000000u : 0u;
	if (flops < 2e8) launch_pdl(cfg, k_gemm_z, tiles, outs, cons, splits, counters, a, b, o, w, fa, fb);
	else CTG_CUDA(cudaLaunchKernelEx(&cfg, k_gemm_z, tiles, outs, cons, splits, counters, a, b, o, w, fa, fb));
}

// ------------------------------------------------------------------------------------
// block permutation (dense_tensor_transpose, dense_tensor.c:799-932)
// ------------------------------------------------------------------------------------

// Permutations and row maps move one to three megabytes of small blocks: bound by latency (chunk, descriptor,
// source, result) and by the integer divisions of the index arithmetic. The descriptor, which belongs to
// the plan, goes to shared memory before the wait on the kernel before, and a thread takes COPY_BATCH
// entries at a time, their divisions and loads side by side. Hubbard chain at D = 256, per launch: permutations
// 11.6 -> 6.9 us, row maps 6.4 -> 4.5; the two-site search 251 -> 248.5 ms, the one-site search 59.5 -> 57.7, energy and
// norm 4.45 -> 4.2. Chunks of 1024 instead of 4096 entries: 5.8 and 3.7 us, the searches within their noise.
// the block's descriptor to shared memory, by all threads
template <class D>
__device__ __forceinline__ void copy_desc(D* to, const D* __restrict__ from)
{
	static_assert(sizeof(D) % sizeof(int) == 0, "descriptors are whole words");
	for (int i = threadIdx.x; i < (int)(sizeof(D) / sizeof(int)); i += blockDim.x) ((int*)to)[i] = ((const int*)from)[i];
	__syncthreads();
}

// T = double, or double2 for complex128 entries (same descriptors, element units)
template <class T>
__global__ void __launch_bounds__(256)
k_permute(const Chunk* __restrict__ chunks, const PermDesc* __restrict__ descs, const T* src, T* dst)
{
	__shared__ PermDesc d;
	const Chunk ch = chunks[blockIdx.x];
	copy_desc(&d, descs + ch.desc);
	pdl_wait();
	pdl_trigger();
	const i64 end = min(d.n, ch.start + (i64)COPY_CHUNK);
	if (d.n < ((i64)1 << 31))
	{
		// 32-bit index arithmetic (64-bit integer division is several times slower)
		const int nd = d.ndim;
		const T* s = src + d.src_off;
		T* t = dst + d.dst_off;
		for (unsigned e0 = copy_first(ch.start, threadIdx.x); e0 < (unsigned)end; e0 = copy_next(e0, blockDim.x))
		{
			unsigned r[COPY_BATCH];
			i64 so[COPY_BATCH];
			T v[COPY_BATCH];
#pragma unroll
			for (int u = 0; u < COPY_BATCH; u++)
			{
				r[u] = copy_entry(e0, u, blockDim.x);
				so[u] = 0;
			}
			for (int i = nd - 1; i > 0; i--)
			{
				const unsigned di = (unsigned)d.dims[i];
				const i64 st = d.sstr[i];
#pragma unroll
				for (int u = 0; u < COPY_BATCH; u++)
				{
					const unsigned q = r[u] / di;
					so[u] += (i64)(r[u] - q * di) * st;
					r[u] = q;
				}
			}
			const i64 st0 = d.sstr[0];
#pragma unroll
			for (int u = 0; u < COPY_BATCH; u++)
				if (copy_entry(e0, u, blockDim.x) < (unsigned)end) v[u] = s[so[u] + (i64)r[u] * st0];
#pragma unroll
			for (int u = 0; u < COPY_BATCH; u++)
				if (copy_entry(e0, u, blockDim.x) < (unsigned)end) t[copy_entry(e0, u, blockDim.x)] = v[u];
		}
		return;
	}
	for (i64 e = ch.start + threadIdx.x; e < end; e += blockDim.x)
	{
		i64 r = e, so = 0;
		for (int i = d.ndim - 1; i >= 0; i--)
		{
			const i64 q = r / d.dims[i];
			so += (r - q * d.dims[i]) * d.sstr[i];
			r = q;
		}
		dst[d.dst_off + e] = src[d.src_off + so];
	}
}

void launch_permute(int nchunks, const Chunk* chunks, const PermDesc* descs, const double* src, double* dst, cudaStream_t st,
                    bool cplx)
{
	if (nchunks <= 0) return;
	const cudaLaunchConfig_t cfg = launch_config(dim3(nchunks), dim3(256), 0, st);
	if (cplx) launch_pdl(cfg, k_permute<double2>, chunks, descs, (const double2*)src, (double2*)dst);
	else launch_pdl(cfg, k_permute<double>, chunks, descs, src, dst);
	CTG_CUDA(cudaGetLastError());
}

// ------------------------------------------------------------------------------------
// row maps: flatten / split / slice (block_sparse_tensor.c:950-1553)
// ------------------------------------------------------------------------------------

template <class T>
__global__ void __launch_bounds__(256)
k_rowmap(const Chunk* __restrict__ chunks, const RowDesc* __restrict__ descs, const i64* __restrict__ maps, const T* src, T* dst)
{
	__shared__ RowDesc d;
	const Chunk ch = chunks[blockIdx.x];
	copy_desc(&d, descs + ch.desc);
	pdl_wait();
	pdl_trigger();
	const i64 n = d.nlead * d.nrow * d.ntrail;
	const i64 end = min(n, ch.start + (i64)COPY_CHUNK);
	const i64* map = maps + d.map_off;
	if (n < ((i64)1 << 31))
	{
		// 32-bit index arithmetic (64-bit integer division is several times slower)
		const unsigned nt = (unsigned)d.ntrail, nr = (unsigned)d.nrow;
		const bool scatter = d.scatter != 0;
		const i64 srows = d.src_rows, drows = d.dst_rows;
		const T* s = src + d.src_off;
		T* o = dst + d.dst_off;
		for (unsigned e0 = copy_first(ch.start, threadIdx.x); e0 < (unsigned)end; e0 = copy_next(e0, blockDim.x))
		{
			unsigned t[COPY_BATCH], lead[COPY_BATCH], j[COPY_BATCH];
			i64 mj[COPY_BATCH];
			T v[COPY_BATCH];
#pragma unroll
			for (int u = 0; u < COPY_BATCH; u++)
			{
				const unsigned e = copy_entry(e0, u, blockDim.x);
				const unsigned lj = e / nt;
				t[u] = e - lj * nt;
				lead[u] = lj / nr;
				j[u] = lj - lead[u] * nr;
				if (e < (unsigned)end) mj[u] = map[j[u]];
			}
#pragma unroll
			for (int u = 0; u < COPY_BATCH; u++)
				if (copy_entry(e0, u, blockDim.x) < (unsigned)end)
					v[u] = s[((i64)lead[u] * srows + (scatter ? (i64)j[u] : mj[u])) * nt + t[u]];
#pragma unroll
			for (int u = 0; u < COPY_BATCH; u++)
				if (copy_entry(e0, u, blockDim.x) < (unsigned)end)
					o[((i64)lead[u] * drows + (scatter ? mj[u] : (i64)j[u])) * nt + t[u]] = v[u];
		}
		return;
	}
	for (i64 e = ch.start + threadIdx.x; e < end; e += blockDim.x)
	{
		const i64 t = e % d.ntrail;
		const i64 lj = e / d.ntrail;
		const i64 j = lj % d.nrow;
		const i64 lead = lj / d.nrow;
		const i64 mj = map[j];
		const i64 srow = d.scatter ? j : mj;
		const i64 drow = d.scatter ? mj : j;
		dst[d.dst_off + (lead * d.dst_rows + drow) * d.ntrail + t] = src[d.src_off + (lead * d.src_rows + srow) * d.ntrail + t];
	}
}

void launch_rowmap(int nchunks, const Chunk* chunks, const RowDesc* descs, const i64* maps, const double* src, double* dst,
                   cudaStream_t st, bool cplx)
{
	if (nchunks <= 0) return;
	const cudaLaunchConfig_t cfg = launch_config(dim3(nchunks), dim3(256), 0, st);
	if (cplx) launch_pdl(cfg, k_rowmap<double2>, chunks, descs, maps, (const double2*)src, (double2*)dst);
	else launch_pdl(cfg, k_rowmap<double>, chunks, descs, maps, src, dst);
	CTG_CUDA(cudaGetLastError());
}

// ------------------------------------------------------------------------------------
// pointwise multiplication along an axis (block_sparse_tensor_multiply_pointwise_vector,
// block_sparse_tensor.c:1654-1703)
// ------------------------------------------------------------------------------------

__device__ __forceinline__ double scale_entry(double x, double f) { return x * f; }
__device__ __forceinline__ double2 scale_entry(double2 x, double f) { return make_double2(x.x * f, x.y * f); }

template <class T>
__global__ void __launch_bounds__(256)
k_scale_axis(const Chunk* __restrict__ chunks, const ScaleDesc* __restrict__ descs, const i64* __restrict__ maps,
             const double* __restrict__ vec, const T* __restrict__ src, T* __restrict__ dst)
{
	pdl_wait();
	pdl_trigger();
	const Chunk ch = chunks[blockIdx.x];
	const ScaleDesc d = descs[ch.desc];
	const i64 n = d.nlead * d.nax * d.ntrail;
	const i64 end = min(n, ch.start + (i64)COPY_CHUNK);
	if (n < ((i64)1 << 31))
	{
		const unsigned nt = (unsigned)d.ntrail, na = (unsigned)d.nax;
		for (unsigned e = (unsigned)ch.start + threadIdx.x; e < (unsigned)end; e += blockDim.x)
		{
			const unsigned q = e / nt;
			const unsigned p = q - (q / na) * na;
			dst[d.off + e] = scale_entry(src[d.off + e], vec[maps[d.map_off + p]]);
		}
		return;
	}
	for (i64 e = ch.start + threadIdx.x; e < end; e += blockDim.x)
	{
		const i64 p = (e / d.ntrail) % d.nax;
		dst[d.off + e] = scale_entry(src[d.off + e], vec[maps[d.map_off + p]]);
	}
}

void launch_scale_axis(int nchunks, const Chunk* chunks, const ScaleDesc* descs, const i64* maps, const double* vec,
                       const double* src, double* dst, cudaStream_t st, bool cplx)
{
	if (nchunks <= 0) return;
	const cudaLaunchConfig_t cfg = launch_config(dim3(nchunks), dim3(256), 0, st);
	if (cplx) launch_pdl(cfg, k_scale_axis<double2>, chunks, descs, maps, vec, (const double2*)src, (double2*)dst);
	else launch_pdl(cfg, k_scale_axis<double>, chunks, descs, maps, vec, src, dst);
	CTG_CUDA(cudaGetLastError());
}

// ------------------------------------------------------------------------------------
// FP64 FMA throughput probe: the denominator of the plain path's roofline
// ------------------------------------------------------------------------------------

__global__ void __launch_bounds__(256) k_fp64_fma(double* out, int iters, double a, double b)
{
	double x[8];
#pragma unroll
	for (int i = 0; i < 8; i++) x[i] = threadIdx.x * 1e-9 + i;
	for (int it = 0; it < iters; it++)
	{
#pragma unroll
		for (int i = 0; i < 8; i++) x[i] = fma(x[i], a, b);
	}
	double s = 0;
#pragma unroll
	for (int i = 0; i < 8; i++) s += x[i];
	if (s == 12345.678) out[0] = s;   // keeps the chains alive
}

double measure_fp64_fma_tflops(int device)
{
	CTG_CUDA(cudaSetDevice(device));
	int sms = 0;
	CTG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
	double* out = nullptr;
	CTG_CUDA(cudaMalloc(&out, sizeof(double)));
	cudaEvent_t e0, e1;
	CTG_CUDA(cudaEventCreate(&e0));
	CTG_CUDA(cudaEventCreate(&e1));
	const int blocks = sms * 8, threads = 256, iters = 4096;
	k_fp64_fma<<<blocks, threads>>>(out, 64, 0.999999, 1e-7);
	CTG_CUDA(cudaEventRecord(e0));
	for (int r = 0; r < 5; r++) k_fp64_fma<<<blocks, threads>>>(out, iters, 0.999999, 1e-7);
	CTG_CUDA(cudaEventRecord(e1));
	CTG_CUDA(cudaEventSynchronize(e1));
	float ms = 0;
	CTG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	cudaFree(out);
	const double flops = 5.0 * blocks * threads * (double)iters * 8 * 2;
	return flops / (ms * 1e-3) / 1e12;
}

}  // namespace ctg
