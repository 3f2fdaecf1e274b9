// soft64.cuh -- double-precision products of the plain FP64 form on the
// integer pipes.
//
// GB300 issues one FP64 warp instruction every 64 cycles and scheduler
// partition, a 32 x 32 -> 64 bit multiply-add (mad.wide) every 2 and a
// 64-bit shift every 4 (measured, four warps per partition).  A product sum
// sum_k P[i][k] x[k] of four positive terms therefore costs 256 cycles as
// four FMAs and about 50 as integers:
//
//   - a positive normal double is M 2^(E - 1085) with M its 53-bit
//     significand shifted left by 10 (2^62 <= M < 2^63) and E its biased
//     exponent;
//   - the upper 64 bits of a product of two such M take three mad.wide
//     (2^60 <= prod < 2^62, at most two units too small);
//   - terms are aligned to the largest exponent sum of the row, each shifted
//     right by its own distance, and added as 64-bit integers;
//   - the sum S (2^60 <= S < 2^64) keeps its exponent, so the two children's
//     sums multiply and round to a double once.
//
// (Of a node's four states the walk leaves one to the FP64 pipe, which would
// otherwise idle.)
//
// A term keeps at least 60 significant bits relative to the row's largest
// term and nothing rounds in between, so a node's value is within 0.6 units
// in the last place of the exact product of sums (four chained FMAs, then a
// product: up to about four).  Everything here expects positive normal
// numbers; `plain` tables, other inputs (zero, negative, subnormal,
// infinite, NaN) and results outside the normal range go through FP64
// instructions instead (the caller's job).
//
// Compiles for the host too, where the arithmetic is tested.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define B3G_HD __host__ __device__ __forceinline__
#else
#define B3G_HD inline
#endif

namespace b3g {

// Transition table of one (entry, side, category): row k holds P[0][k] as a
// double and the significands and biased exponents of P[i][k], i = 1..3; row
// 4 is the unknown state (all ones).  State 0 stays with the FP64 pipe, which
// works beside the integer pipes: a quarter of the products costs it 256
// cycles a sum, less than the integer pipes take for the other three.
struct SoftRow4 {
	uint32_t hi[3], lo1; // hi of i = 1, 2, 3; lo of i = 1
	uint32_t lo2, lo3;
	double d0;
};
struct SoftTab4 {
	SoftRow4 row[5];
	uint32_t e[5][2]; // exponents of i = 1 (low half) and 2 (high), of i = 3
	uint32_t plain;   // some entry is not a positive normal number
	uint32_t pad;
};
static_assert(sizeof(SoftTab4) == 208, "13 copies of 16 bytes");

constexpr int32_t kSoftBias = 1085;         // value = M 2^(E - 1085)
constexpr int32_t kSoftDotBias = 2106;      // sum of products: S 2^(m - 2106)

struct SoftNum {
	uint32_t hi, lo;
	uint32_t e; // biased exponent, 1..2046
};

// True when the high word is that of a positive normal double.
B3G_HD bool soft_normal(uint32_t dhi)
{
	return dhi - 0x00100000u < 0x7FE00000u;
}

B3G_HD SoftNum soft_split(uint32_t dhi, uint32_t dlo)
{
	SoftNum r;
	r.hi = (((dhi & 0xFFFFFu) | 0x100000u) << 10) | (dlo >> 22);
	r.lo = dlo << 10;
	r.e = dhi >> 20;
	return r;
}

// Upper 64 bits of the product of two significands (at most two units low).
B3G_HD uint64_t soft_prod(uint32_t xh, uint32_t xl, uint32_t ph, uint32_t pl)
{
	// xh, ph < 2^31: the cross terms' sum stays below 2^64
	const uint64_t t = (uint64_t)xl * ph + (uint64_t)xh * pl;
	return (uint64_t)xh * ph + (t >> 32);
}

// 64-bit right shift by d (0 for d >= 64).
B3G_HD uint64_t soft_shr(uint64_t v, uint32_t d)
{
#ifdef __CUDA_ARCH__
	uint64_t r;
	asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(d));
	return r;
#else
	return d >= 64 ? 0 : v >> d;
#endif
}

// Largest of two pairs of 16-bit halves.
B3G_HD uint32_t soft_max2(uint32_t a, uint32_t b)
{
#ifdef __CUDA_ARCH__
	uint32_t r;
	asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
	return r;
#else
	const uint32_t al = a & 0xFFFFu, bl = b & 0xFFFFu, ah = a >> 16, bh = b >> 16;
	return (al > bl ? al : bl) | ((ah > bh ? ah : bh) << 16);
#endif
}

B3G_HD int soft_clz(uint32_t x)
{
#ifdef __CUDA_ARCH__
	return __clz((int)x);
#else
	return x ? __builtin_clz(x) : 32;
#endif
}

// Product of two nonzero 64-bit significands a 2^ea and b 2^eb (top bits no
// lower than bit 60), rounded to a double's bits.  ok: the exponent lies
// well inside the normal range (otherwise the result is meaningless).
B3G_HD uint64_t soft_mul_round(uint64_t a, int32_t ea, uint64_t b, int32_t eb, bool &ok)
{
	const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a;
	const uint32_t bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
	const uint64_t q1 = (uint64_t)al * bh;
	const uint64_t q2 = (uint64_t)ah * bl + (uint32_t)q1;
	uint64_t h = (uint64_t)ah * bh + (q1 >> 32) + (q2 >> 32); // >= 2^56
	const int lz = soft_clz((uint32_t)(h >> 32));             // 0..7
	h <<= lz;
	const int32_t eb2 = ea + eb + 1150 - lz; // biased exponent before rounding
	ok = eb2 >= 1 && eb2 <= 2045;
	const uint64_t mant = (h >> 11) + ((h >> 10) & 1u);
	// the significand's leading one adds the missing 1 to the exponent; a
	// rounding carry adds another
	return mant + ((uint64_t)(uint32_t)(eb2 - 1) << 52);
}

// The product of a positive normal double's bits and the positive normal
// number `f`, rounded; the exponent of the result must lie in the normal
// range (a caller that scales a small number up to at most 1 knows it does).
B3G_HD uint64_t soft_scale(uint64_t bits, const SoftNum &f)
{
	const SoftNum n = soft_split((uint32_t)(bits >> 32), (uint32_t)bits);
	const uint64_t p = soft_prod(n.hi, n.lo, f.hi, f.lo); // 2^60 <= p < 2^62
	const uint32_t s = (uint32_t)(p >> 61);
	const uint64_t q = p >> s; // 2^60 <= q < 2^61
	const uint64_t mant = (q >> 8) + ((q >> 7) & 1u);
	return mant + ((uint64_t)(n.e + f.e - 1024u + s) << 52);
}

} // namespace b3g
