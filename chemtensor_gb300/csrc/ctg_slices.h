// ctg_slices.h - exact digit slices of FP64 numbers, for block products on the FP16 / BF16 tensor cores.
//
// Every row of an operand of a product gets one power of two 2^e above all of its entries. An entry x
// becomes the 64-bit fixed-point number v = x 2^(62 - e) (|v| <= 2^62; digits of x below 2^(e - 62) are
// cut off) and v is written in base 256 with balanced digits, v = sum_s d_s 2^(56 - 8 s), s = 0 .. 7,
// -128 <= d_s <= 127. A digit is exact in FP16 and BF16, a product of two digits and sums of up to
// 2^24 / (8 * 2^14) = 128 terms of one order s + t are exact in FP32, so the tensor cores form
//   acc_o = sum_{s + t = o} sum_k d_s(k) d'_t(k),  o = 0 .. 7
// without any rounding, and sum_k x(k) y(k) = 2^(e + f - 68) sum_o acc_o 2^(56 - 8 o) up to the orders
// o >= 8, which lie below 2^-59 2^(e + f) for each term (2^-62 in the root mean square) (the error-free
// splitting of K. Ozaki, T. Ogita, S. Oishi, S. M. Rump, Numer. Algorithms 59, 2012, with integer digits).
// The sum over o is an integer, accumulated over the whole contraction and rounded once.
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

namespace ctg {

constexpr int SLICES = 8;                  // digits of an entry
constexpr int SLICE_K = 128;               // terms summed in FP32 before the sums move to integers
constexpr int SLICE_TERMS_MAX = 1 << 21;   // most terms of a result: its low orders, below 2^48 per 128 terms, stay in 63 bits
constexpr int SLICE_EXP_MIN = 128;         // rows whose largest entry has a smaller biased exponent (or holds a
                                           // number that is not finite) are summed in FP64 instead
constexpr int SLICE_EXP_ZERO = -4000;      // in place of the exponent: a row of zeros
constexpr int SLICE_EXP_FP64 = 20000;      // a row that is summed in FP64
constexpr uint64_t SLICE_BIAS = 0x8080808080808080ull;

// magnitude of the number with the bits (hi, lo) in a row whose largest biased exponent is
// E >= SLICE_EXP_MIN (a row of zeros takes any such E), as biased digits: d_s + 128 in byte 7 - s. The
// number's sign turns all of its digits.
__host__ __device__ inline uint64_t slice_digits(uint32_t hi, uint32_t lo, int E)
{
	// the hidden bit that zeros and denormal numbers do not have is shifted out: E - 0 > 62
	const uint64_t m = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
	int d = E - (int)((hi >> 20) & 0x7ff);
	d = d > 63 ? 63 : d;
	return ((m << 9) >> d) + SLICE_BIAS;
}

// Biased exponent of a sum whose 96-bit magnitude has its leading bit at the top, for two rows with the
// biased exponents E and F; slice_value subtracts the leading zeros. Every result of the two rows lies in
// the normal range if slice_in_range.
__host__ __device__ inline int slice_top(int E, int F) { return E + F - 2112 + 1023 + 95; }
__host__ __device__ inline bool slice_in_range(int top) { return top - 96 >= 1 && top + 1 <= 2046; }

// the exponent of a row as the product reads it, from its largest biased exponent (0: zeros only, 1: denormal
// numbers at most, 0x7ff: a number that is not finite)
__host__ __device__ inline int slice_exp(int code)
{
	return code == 0 ? SLICE_EXP_ZERO : code < SLICE_EXP_MIN || code == 0x7ff ? SLICE_EXP_FP64 : code;
}

// The digits that are cut off (2^-62, and the orders o >= 8, 2^-59.2 at most, 2^-62.2 in the root mean square, of
// 2^(e + f) for each term) lie within the rounding of an FP64 sum if some term is not much smaller than the product
// of its rows' largest entries: if the biased exponents of its factors add up to slice_term_limit at least, k
// terms are off by sqrt(k) 2^-53.2 of that term (k 2^-50.2 for the worst digits), an FP64 sum by up to k 2^-53 of
// the sum of all magnitudes.
constexpr int SLICE_TERM = 7;
__host__ __device__ inline int slice_term_limit(int e, int f) { return e + f - SLICE_TERM; }

// Whether a result with the biased exponent r of two rows with these exponents has to be looked at again: it may
// leave the normal range, a row is not finite or tiny, or the result is so small that it does not itself show
// that it has such a term. That of a row of zeros only if it meets a row that is not finite (NaN) or tiny.
__host__ __device__ inline bool slice_suspect(int e, int f, int r)
{
	return e + f >= SLICE_EXP_ZERO / 2 && (!slice_in_range(slice_top(e, f)) || r < slice_term_limit(e, f) - 1023);
}

// bits of the FP64 number nearest to (h 2^32 + l) 2^(E + F - 2112) (ties away from zero), the value of a
// sum over the orders with weights 2^(56 - 8 o): h the orders 0 .. 3 (units of 2^32), l the orders 4 .. 7,
// top = slice_top(E, F)
__host__ __device__ inline uint64_t slice_value(int64_t h, int64_t l, int top)
{
	h += l >> 32;
	uint32_t w0 = (uint32_t)l, w1 = (uint32_t)h, w2 = (uint32_t)((uint64_t)h >> 32);
	const uint32_t sign = w2 & 0x80000000u;
	if (sign)
	{
		// negate the 96-bit number
		w0 = 0u - w0;
		const uint64_t n = ~(uint64_t)h + (w0 == 0 ? 1 : 0);
		w1 = (uint32_t)n;
		w2 = (uint32_t)(n >> 32);
	}
	if (w2 == 0)
	{
		w2 = w1;
		w1 = w0;
		w0 = 0;
		top -= 32;
	}
	if (w2 == 0)
	{
		w2 = w1;
		w1 = 0;
		top -= 32;
	}
#ifdef __CUDA_ARCH__
	const int lz = __clz((int)w2);
	const uint32_t m1 = __funnelshift_l(w1, w2, lz), m0 = __funnelshift_l(w0, w1, lz);
#else
	const int lz = w2 ? __builtin_clz(w2) : 32;
	const uint32_t m1 = lz == 0 || lz == 32 ? w2 : (w2 << lz) | (w1 >> (32 - lz));
	const uint32_t m0 = lz == 0 || lz == 32 ? w1 : (w1 << lz) | (w0 >> (32 - lz));
#endif
	if (w2 == 0) return 0;
	// 53 bits with the leading one added into the exponent field, so that a carry of the rounding moves on
	const uint64_t m = ((uint64_t)m1 << 32) | m0;
	const uint64_t e = (uint64_t)((uint32_t)(top - lz - 1) << 20 | sign) << 32;
	return e + (m >> 11) + ((m0 >> 10) & 1);
}

}  // namespace ctg
