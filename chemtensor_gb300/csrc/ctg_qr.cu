// ctg_qr.cu - QR / RQ of each block by Householder reflections, double and complex128 entries.
//
// QR (desc.qr = 1) follows LAPACK's geqrf + orgqr / ungqr in dense_tensor_qr_fill (dense_tensor.c:2253-2651):
// A = Q R, R upper triangular with real diagonal entries -sign(Re alpha) |x| of the reflectors (alpha itself
// where there is nothing below it to eliminate).
// RQ (desc.qr = 0) follows gerqf + orgrq / ungrq in dense_tensor_rq_fill (dense_tensor.c:2680-2880): gerqf
// eliminates the rows of A from the last one upwards, each towards its trailing column; that is the QR
// above applied to W = J A^H J (J reverses an index), with A = (J R_W^H J) (J Q_W^H J).
//
// One CTA per block, W (p x s) column-major in shared memory where it fits, else in the block's scratch.
// Bound by the serial chain over the columns and by the FP64 instructions of one SM: each occupies its
// sub-partition for 64 cycles. Hence
//   - v = (alpha - beta, x) as it stands, H^H = I - f v v^H with f = conj(tau) / |alpha - beta|^2: no pass that
//     scales x, and the last warp derives f from |x|^2 while the others already form x^H b for their
//     columns; two barriers per column;
//   - a warp takes two columns at a time and adds their sums in the same exchanges (five adds for two real
//     columns, six for two complex ones, instead of ten and twenty);
//   - square root and reciprocals by ctg_fp64.cuh, an FP64 division takes a thousand cycles;
//   - Q replaces the reflectors in place, column c from H_c on, columns c.. only: one barrier per column.
// One-site search of a Hubbard chain at D = 256: 131 -> 83 us per call, the search 68.8 -> 60.2 ms; complex entries at
// D = 64 211 -> 37 us. (Before: one warp per column with a reduction each, matrix in global memory, three to
// four barriers and FP64 divisions per column, Q over all columns.)
#include <algorithm>
#include <cfloat>
#include <climits>

#include "ctg_fp64.cuh"
#include "ctg_kernels.h"

namespace ctg {

namespace {

constexpr int QR_THREADS = 512;
constexpr int QR_WARPS = QR_THREADS / 32;
constexpr int QR_PAIRS = 4;                       // column pairs of a warp between two barriers
constexpr int QR_SMEM_LIMIT = 200 * 1024;

__host__ __device__ inline i64 qr_entries(i64 p, i64 s, i64 k) { return p * s + 2 * k; }

__device__ __forceinline__ double conj_of(double a) { return a; }
__device__ __forceinline__ double2 conj_of(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double mul(double a, double b) { return a * b; }
__device__ __forceinline__ double2 mul(double2 a, double2 b)
{
	return make_double2(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}
// s += conj(x) b. Complex products are rounded by themselves and then added: one rounding of the size of the
// sum (or of b) instead of two
__device__ __forceinline__ void add_dot(double& s, double x, double b) { s = fma(x, b, s); }
__device__ __forceinline__ void add_dot(double2& s, double2 x, double2 b)
{
	s.x += fma(x.x, b.x, x.y * b.y);
	s.y += fma(x.x, b.y, -(x.y * b.x));
}
// b - t x
__device__ __forceinline__ double sub_mul(double b, double t, double x) { return fma(-t, x, b); }
__device__ __forceinline__ double2 sub_mul(double2 b, double2 t, double2 x)
{
	return make_double2(b.x - fma(t.x, x.x, -(t.y * x.y)), b.y - fma(t.x, x.y, t.y * x.x));
}
__device__ __forceinline__ double abs2(double x, double s) { return fma(x, x, s); }
__device__ __forceinline__ double abs2(double2 x, double s) { return fma(x.x, x.x, fma(x.y, x.y, s)); }
__device__ __forceinline__ double scaled(double x, double f) { return x * f; }
__device__ __forceinline__ double2 scaled(double2 x, double f) { return make_double2(x.x * f, x.y * f); }
__device__ __forceinline__ double one_of(double) { return 1.0; }
__device__ __forceinline__ double2 one_of(double2) { return make_double2(1.0, 0.0); }
__device__ __forceinline__ int abs_hi(double x) { return __double2hiint(x) & 0x7fffffff; }
__device__ __forceinline__ int abs_hi(double2 x) { return max(abs_hi(x.x), abs_hi(x.y)); }

// both sums over the warp, to every lane; each exchange hands half of what is left over
__device__ __forceinline__ void warp_sums(double& a, double& b)
{
	const bool hi = threadIdx.x & 16;
	double c = (hi ? b : a) + __shfl_xor_sync(0xffffffffu, hi ? a : b, 16);
#pragma unroll
	for (int o = 8; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
	a = __shfl_sync(0xffffffffu, c, 0);
	b = __shfl_sync(0xffffffffu, c, 16);
}
__device__ __forceinline__ void warp_sums(double2& a, double2& b)
{
	const bool hi = threadIdx.x & 16, odd = threadIdx.x & 8;
	const double c = (hi ? b.x : a.x) + __shfl_xor_sync(0xffffffffu, hi ? a.x : b.x, 16);
	const double d = (hi ? b.y : a.y) + __shfl_xor_sync(0xffffffffu, hi ? a.y : b.y, 16);
	double e = (odd ? d : c) + __shfl_xor_sync(0xffffffffu, odd ? c : d, 8);
#pragma unroll
	for (int o = 4; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
	a.x = __shfl_sync(0xffffffffu, e, 0);
	a.y = __shfl_sync(0xffffffffu, e, 8);
	b.x = __shfl_sync(0xffffffffu, e, 16);
	b.y = __shfl_sync(0xffffffffu, e, 24);
}
__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
	return v;
}

// The reflector of (alpha, x), xn2 = |x|^2: H^H (alpha, x) = (beta, 0), H^H = I - f v v^H, v = (v0, x). f = 0: H = I.
// H is as orthogonal as f is accurate for the v0 that is used, rounding and all: f = 2 / (v0^2 + xn2), and for complex
// entries f = 2 Re v0 conj(v0) / (|v0|^2 (|v0|^2 + xn2)), whose five roundings would make it 1.5 times as far off as
// LAPACK's scaled vectors and which is therefore formed in pairs of numbers (after an exact scaling that keeps
// the products in range).
// Squared norms below 1e-306 (of a block whose entries lie in a normal range) are zeros to all purposes: f,
// their reciprocal, must stay a number. The functions of ctg_fp64.cuh want normal numbers and their
// reciprocals: squared norms beyond 1e-290 and 1e290, infinities and NaN (which stay NaN in the factors, as
// in LAPACK) take the IEEE operations.
__device__ __forceinline__ bool plain_range(double n2) { return n2 > 1e-290 && n2 < 1e290; }
__device__ __noinline__ double ieee_sqrt(double x) { return sqrt(x); }
__device__ __noinline__ double ieee_rcp(double x) { return 1.0 / x; }
__device__ __forceinline__ void reflector(double alpha, double xn2, double& beta, double& v0, double& f)
{
	const double n2 = fma(alpha, alpha, xn2);
	beta = alpha;
	v0 = f = 0.0;
	if (xn2 == 0.0 || n2 <= 1e-306) return;
	const bool plain = plain_range(n2);
	beta = -copysign(plain ? sqrt64(n2) : ieee_sqrt(n2), alpha);
	v0 = alpha - beta;
	const double d = fma(v0, v0, xn2);
	f = 2.0 * (plain ? rcp64(d) : ieee_rcp(d));
}
__device__ __forceinline__ void reflector(double2 alpha, double xn2, double& beta, double2& v0, double2& f)
{
	const double n2 = abs2(alpha, xn2);
	beta = alpha.x;
	v0 = f = make_double2(0.0, 0.0);
	if ((xn2 == 0.0 && alpha.y == 0.0) || n2 <= 1e-306) return;
	const bool plain = plain_range(n2);
	beta = -copysign(plain ? sqrt64(n2) : ieee_sqrt(n2), alpha.x);
	v0 = make_double2(alpha.x - beta, alpha.y);
	if (!(n2 <= DBL_MAX))
	{
		f.x = f.y = 0.0 * n2;
		return;
	}
	// |Re v0| is the largest of the entries' magnitudes, up to a factor: scaled to [1, 2)
	const double sc = __hiloint2double((2046 - ((__double2hiint(v0.x) >> 20) & 0x7ff)) << 20, 0);
	const double vx = v0.x * sc, vy = v0.y * sc;
	// |v0|^2 = a + al, |v0|^2 + xn2 = b + bl
	const double p = vx * vx, pe = fma(vx, vx, -p), q = vy * vy, qe = fma(vy, vy, -q);
	const double a = p + q, al = (q - (a - p)) + (pe + qe);              // p >= q
	const double x2 = xn2 * sc * sc, b = a + x2, bb = b - a;
	const double bl = ((a - (b - bb)) + (x2 - bb)) + al;
	// 1 / ((a + al) (b + bl)) = y + yl
	const double y = rcp64(a * b), t = a * y, te = fma(a, y, -t);
	double r = fma(-b, t, 1.0);
	r = fma(-b, te, r);
	r = fma(-bl, t, r);
	r = fma(-b * al, y, r);
	const double yl = y * r;
	const double m = vx * vy, me = fma(vx, vy, -m), s2 = 2.0 * sc;
	f.x = s2 * (fma(p, y, fma(p, yl, pe * y)) * sc);
	f.y = -s2 * (fma(m, y, fma(m, yl, me * y)) * sc);
}

template <class T>
__global__ void __launch_bounds__(QR_THREADS, 1)
k_qr_householder(const RqDesc* __restrict__ descs, const T* __restrict__ a, T* __restrict__ r, T* __restrict__ q,
                 T* __restrict__ scratch, int smem_bytes)
{
	extern __shared__ __align__(16) unsigned char qr_sm[];
	__shared__ T sh_f, sh_v0;
	__shared__ int red[QR_WARPS];
	const RqDesc d = descs[blockIdx.x];
	const int m = d.m, n = d.n;
	const bool qr = d.qr != 0;
	const int k = min(m, n);
	const int p = qr ? m : n, s = qr ? n : m;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	T* B = qr_entries(p, s, k) * (i64)sizeof(T) <= smem_bytes ? (T*)qr_sm : scratch + d.w_off;
	T* F = B + (i64)p * s;                      // k: the reflectors' factors
	double* beta = (double*)(F + k);            // k: the diagonal of R_W
	const T* ab = a + d.a_off;
	int big = 0;
	for (i64 e = tid; e < (i64)p * s; e += QR_THREADS)
	{
		const i64 i = e % p, j = e / p;
		const T x = qr ? ab[i * n + j] : conj_of(ab[(m - 1 - j) * n + (n - 1 - i)]);
		B[e] = x;
		big = max(big, abs_hi(x));
	}
	big = __reduce_max_sync(0xffffffffu, big);
	if (lane == 0) red[warp] = big;
	__syncthreads();
	for (int w = 0; w < QR_WARPS; w++) big = max(big, red[w]);
	// a block of extreme scale is brought to entries around 1, exactly
	int ex = (big >> 20) - 1023;
	if (big >= 0x7ff00000 || big == 0 || (ex > -100 && ex < 100)) ex = 0;
	ex = max(ex, -1000);
	if (ex != 0)
	{
		const double sc = scalbn(1.0, -ex);
		for (i64 e = tid; e < (i64)p * s; e += QR_THREADS) B[e] = scaled(B[e], sc);
		__syncthreads();
	}
	for (int c = 0; c < k; c++)
	{
		T* x = B + (i64)c * p;
		if (warp == QR_WARPS - 1)
		{
			double xn2 = 0;
			for (int i = c + 1 + lane; i < p; i += 32) xn2 = abs2(x[i], xn2);
			xn2 = warp_sum(xn2);
			double be;
			T v0, f;
			reflector(x[c], xn2, be, v0, f);
			__syncwarp();
			if (lane == 0)
			{
				sh_f = f;
				sh_v0 = v0;
				x[c] = v0;
				F[c] = f;
				beta[c] = be;
			}
		}
		// the pairs of columns right of c: pair g is columns 2 g, 2 g + 1
		const int g0 = (c + 1) >> 1, g1 = (s + 1) >> 1;
		bool first = true;
		for (int gb = g0 + (warp - g0 % QR_WARPS + QR_WARPS) % QR_WARPS; first || gb < g1; gb += QR_WARPS * QR_PAIRS)
		{
			T sum[QR_PAIRS][2];
#pragma unroll
			for (int u = 0; u < QR_PAIRS; u++)
			{
				const int g = gb + u * QR_WARPS;
				sum[u][0] = sum[u][1] = T();
				if (g >= g1) continue;
				const T* b0 = B + (i64)(2 * g) * p;
				const T* b1 = 2 * g + 1 < s ? b0 + p : b0;
				for (int i = c + 1 + lane; i < p; i += 32)
				{
					const T v = x[i];
					add_dot(sum[u][0], v, b0[i]);
					add_dot(sum[u][1], v, b1[i]);
				}
				warp_sums(sum[u][0], sum[u][1]);
			}
			if (first) __syncthreads();             // the factor is there
			first = false;
			const T f = sh_f, v0 = sh_v0;
#pragma unroll
			for (int u = 0; u < QR_PAIRS; u++)
			{
				const int g = gb + u * QR_WARPS;
				if (g >= g1) continue;
				T* b0 = B + (i64)(2 * g) * p;
				T* b1 = b0 + p;
				const bool on0 = 2 * g > c, on1 = 2 * g + 1 < s;
				const T c0 = b0[c], c1 = on1 ? b1[c] : T();
				add_dot(sum[u][0], v0, c0);
				add_dot(sum[u][1], v0, c1);
				const T t0 = mul(f, sum[u][0]), t1 = mul(f, sum[u][1]);
				__syncwarp();
				for (int i = c + 1 + lane; i < p; i += 32)
				{
					const T v = x[i];
					if (on0) b0[i] = sub_mul(b0[i], t0, v);
					if (on1) b1[i] = sub_mul(b1[i], t1, v);
				}
				if (lane == 0)
				{
					if (on0) b0[c] = sub_mul(c0, t0, v0);
					if (on1) b1[c] = sub_mul(c1, t1, v0);
				}
			}
		}
		__syncthreads();
	}
	// R: the upper part of W, beta on the diagonal
	const double us = scalbn(1.0, ex);
	auto r_entry = [&](int i, int j) {            // R_W[i][j]
		T x = T();
		if (i < j) x = B[i + (i64)p * j];
		if (i == j) x = scaled(one_of(T()), beta[i]);
		return ex != 0 ? scaled(x, us) : x;
	};
	if (qr)
		for (i64 e = tid; e < (i64)k * n; e += QR_THREADS) r[d.r_off + e] = r_entry((int)(e / n), (int)(e % n));
	else
		for (i64 e = tid; e < (i64)m * k; e += QR_THREADS)
			r[d.r_off + e] = conj_of(r_entry(k - 1 - (int)(e % k), m - 1 - (int)(e / k)));
	__syncthreads();
	// Q_W = H_0 ... H_{k-1} E in place, backwards: H_c touches rows c.. of columns c.. only
	for (int c = k - 1; c >= 0; c--)
	{
		T* x = B + (i64)c * p;
		const T f = conj_of(F[c]), v0 = x[c];
		const int g0 = (c + 1) >> 1, g1 = (k + 1) >> 1;
		for (int g = g0 + (warp - g0 % QR_WARPS + QR_WARPS) % QR_WARPS; g < g1; g += QR_WARPS)
		{
			T* b0 = B + (i64)(2 * g) * p;
			T* b1 = b0 + p;
			const bool on0 = 2 * g > c, on1 = 2 * g + 1 < k;
			T s0 = T(), s1 = T();
			for (int i = c + 1 + lane; i < p; i += 32)
			{
				const T v = x[i];
				if (on0) add_dot(s0, v, b0[i]);
				if (on1) add_dot(s1, v, b1[i]);
			}
			warp_sums(s0, s1);
			const T t0 = mul(f, s0), t1 = mul(f, s1);
			for (int i = c + 1 + lane; i < p; i += 32)
			{
				const T v = x[i];
				if (on0) b0[i] = sub_mul(b0[i], t0, v);
				if (on1) b1[i] = sub_mul(b1[i], t1, v);
			}
			if (lane == 0)
			{
				if (on0) b0[c] = sub_mul(T(), t0, v0);
				if (on1) b1[c] = sub_mul(T(), t1, v0);
			}
		}
		__syncthreads();                          // nobody reads the reflector any more
		// H_c e_c by the warp that owns the column from now on
		if (warp == (c >> 1) % QR_WARPS)
		{
			const T t = mul(f, conj_of(v0));
			for (int i = lane; i < p; i += 32)
			{
				if (i < c) x[i] = T();
				else if (i == c) x[i] = sub_mul(one_of(T()), t, v0);
				else x[i] = sub_mul(T(), t, x[i]);
			}
			__syncwarp();
		}
	}
	__syncthreads();
	if (qr)
		for (i64 e = tid; e < (i64)m * k; e += QR_THREADS) q[d.q_off + e] = B[e / k + (i64)p * (e % k)];
	else
		for (i64 e = tid; e < (i64)k * n; e += QR_THREADS)
			q[d.q_off + e] = conj_of(B[(n - 1 - e % n) + (i64)p * (k - 1 - e / n)]);
}

// The real QR / RQ whose rounding reduced-precision searches keep (Ctx::steady): matrix in the scratch, scaled
// reflectors, IEEE square roots and divisions, a warp per column. 131 us where the kernel above takes 83.
constexpr int RQ_THREADS = 256;

__device__ double block_sum(double v, double* red)
{
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	v = warp_sum(v);
	__syncthreads();
	if (lane == 0) red[warp] = v;
	__syncthreads();
	double t = 0;
	for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
	return t;
}

__global__ void __launch_bounds__(RQ_THREADS)
k_qr_steady(const RqDesc* __restrict__ descs, const double* __restrict__ a, double* __restrict__ r,
                 double* __restrict__ q, double* __restrict__ scratch)
{
	__shared__ double red[RQ_THREADS / 32];
	__shared__ double sh_beta, sh_tau, sh_scale;
	const RqDesc d = descs[blockIdx.x];
	const int m = d.m, n = d.n;
	const bool qr = d.qr != 0;
	const int k = min(m, n);
	const int p = qr ? m : n, s = qr ? n : m;   // W is p x s, column-major
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = RQ_THREADS / 32;
	double* B = scratch + d.w_off;             // W, p x s
	double* Q = B + (i64)p * s;                // Q_W, p x k
	double* tau = Q + (i64)p * k;              // k
	const double* ab = a + d.a_off;
	for (i64 e = tid; e < (i64)p * s; e += RQ_THREADS)
	{
		const i64 i = e % p, j = e / p;
		B[e] = qr ? ab[i * n + j] : ab[(m - 1 - j) * n + (n - 1 - i)];
	}
	__syncthreads();
	for (int c = 0; c < k; c++)
	{
		double* bc = B + (i64)c * p;
		double part = 0;
		for (int i = c + 1 + tid; i < p; i += RQ_THREADS) part = fma(bc[i], bc[i], part);
		const double xnorm2 = block_sum(part, red);
		if (tid == 0)
		{
			const double alpha = bc[c];
			if (xnorm2 == 0.0)
			{
				sh_tau = 0.0;
				sh_beta = alpha;
				sh_scale = 0.0;
			}
			else
			{
				const double beta = -copysign(sqrt(alpha * alpha + xnorm2), alpha);
				sh_tau = (beta - alpha) / beta;
				sh_beta = beta;
				sh_scale = 1.0 / (alpha - beta);
			}
		}
		__syncthreads();
		const double tc = sh_tau;
		for (int i = c + 1 + tid; i < p; i += RQ_THREADS) bc[i] *= sh_scale;
		__syncthreads();
		if (tid == 0) { bc[c] = sh_beta; tau[c] = tc; }
		__syncthreads();
		// apply H = I - tau v v^T (v = (1, bc[c+1:])) to the remaining columns
		if (tc != 0.0)
		{
			for (int c2 = c + 1 + warp; c2 < s; c2 += nwarps)
			{
				double* b2 = B + (i64)c2 * p;
				double acc = 0;
				for (int i = c + lane; i < p; i += 32) acc = fma(i == c ? 1.0 : bc[i], b2[i], acc);
				acc = warp_sum(acc) * tc;
				for (int i = c + lane; i < p; i += 32) b2[i] -= acc * (i == c ? 1.0 : bc[i]);
			}
		}
		__syncthreads();
	}
	// Q_W = H_0 ... H_{k-1} E (p x k), accumulated backwards, column-major
	for (i64 e = tid; e < (i64)p * k; e += RQ_THREADS) Q[e] = (e / p == e % p) ? 1.0 : 0.0;
	__syncthreads();
	for (int c = k - 1; c >= 0; c--)
	{
		const double tc = tau[c];
		const double* bc = B + (i64)c * p;
		if (tc != 0.0)
		{
			for (int j = warp; j < k; j += nwarps)
			{
				double* qj = Q + (i64)j * p;
				double acc = 0;
				for (int i = c + lane; i < p; i += 32) acc = fma(i == c ? 1.0 : bc[i], qj[i], acc);
				acc = warp_sum(acc) * tc;
				for (int i = c + lane; i < p; i += 32) qj[i] -= acc * (i == c ? 1.0 : bc[i]);
			}
		}
		__syncthreads();
	}
	if (qr)
	{
		// R (k x n) = upper part of W; Q (m x k) = Q_W
		for (i64 e = tid; e < (i64)k * n; e += RQ_THREADS)
		{
			const i64 i = e / n, j = e % n;
			r[d.r_off + e] = (i <= j) ? B[i + (i64)p * j] : 0.0;
		}
		for (i64 e = tid; e < (i64)m * k; e += RQ_THREADS)
		{
			const i64 i = e / k, j = e % k;
			q[d.q_off + e] = Q[i + (i64)p * j];
		}
	}
	else
	{
		// R (m x k): R[i][j] = R_W[k-1-j][m-1-i]; Q (k x n): Q[j][i] = Q_W[n-1-i][k-1-j]
		for (i64 e = tid; e < (i64)m * k; e += RQ_THREADS)
		{
			const i64 i = e / k, j = e % k;
			const i64 a0 = k - 1 - j, b0 = m - 1 - i;
			r[d.r_off + e] = (a0 <= b0) ? B[a0 + (i64)p * b0] : 0.0;
		}
		for (i64 e = tid; e < (i64)k * n; e += RQ_THREADS)
		{
			const i64 j = e / n, i = e % n;
			q[d.q_off + e] = Q[(n - 1 - i) + (i64)p * (k - 1 - j)];
		}
	}
}

template <class T>
void launch_qr_blocks(int nblocks, const RqDesc* descs, const RqDesc* host, const double* a, double* r, double* q,
                      double* scratch, cudaStream_t st)
{
	if (nblocks <= 0) return;
	i64 smem = 0;
	for (int b = 0; b < nblocks; b++)
	{
		const i64 need = qr_entries(host[b].m, host[b].n, std::min(host[b].m, host[b].n)) * (i64)sizeof(T);
		if (need <= QR_SMEM_LIMIT) smem = std::max(smem, need);
	}
	// for every size: the limit that holds without it, 48 KB, counts the kernel's static shared memory too. The
	// attribute belongs to the current device.
	CTG_CUDA(cudaFuncSetAttribute(k_qr_householder<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, QR_SMEM_LIMIT));
	k_qr_householder<T><<<nblocks, QR_THREADS, (size_t)smem, st>>>(descs, (const T*)a, (T*)r, (T*)q, (T*)scratch, (int)smem);
	CTG_CUDA(cudaGetLastError());
}

}  // namespace

void launch_qr(int nblocks, const RqDesc* descs, const RqDesc* host, const double* a, double* r, double* q, double* scratch,
               bool cplx, bool steady, cudaStream_t st)
{
	if (steady && !cplx && nblocks > 0)
	{
		k_qr_steady<<<nblocks, RQ_THREADS, 0, st>>>(descs, a, r, q, scratch);
		CTG_CUDA(cudaGetLastError());
	}
	else if (cplx) launch_qr_blocks<double2>(nblocks, descs, host, a, r, q, scratch, st);
	else launch_qr_blocks<double>(nblocks, descs, host, a, r, q, scratch, st);
}

}  // namespace ctg
