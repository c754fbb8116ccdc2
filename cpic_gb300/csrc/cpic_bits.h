// cpic_bits.h -- exact FP64 conversions done with integer operations on the
// bits of a double.
//
// The FP64 form computes, per particle, the floor of its position in cell
// units (converted to an int cell index) and splits each of its four
// fixed-point deposit values v into hi = rn(v) (the nearest integer, ties to
// even) and lo = rn((v - hi) * 2^m).  In FP64 arithmetic these are FRND,
// F2I, I2F, DADD, DMUL and F2I instructions, all on the FP64 pipe, which is
// narrow on this GPU (about 1.7 instructions per clock per SM, against 64
// for 32-bit integer operations) and is what bounds the FP64 form.  The
// functions below give the same results exactly, bit for bit, from the IEEE
// representation with integer shifts, masks and adds.  They are plain C++
// (host and device), so a CPU test checks them against the FP64 operations
// on edge cases and random values.
#pragma once
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define CPIC_HD __host__ __device__ __forceinline__
#else
#define CPIC_HD inline
#endif

namespace cpic {
namespace bits {

CPIC_HD uint64_t to_bits(double d)
{
#ifdef __CUDA_ARCH__
	// through an asm move: the compiler turns integer tests of a plain
	// bit cast back into FP64 compares (four of them, 80 clocks of an SM per
	// warp, in the fused kernel)
	uint64_t b;
	asm("mov.b64 %0, %1;" : "=l"(b) : "d"(d));
	return b;
#else
	uint64_t b;
	std::memcpy(&b, &d, 8);
	return b;
#endif
}

CPIC_HD double from_bits(uint64_t b)
{
#ifdef __CUDA_ARCH__
	return __longlong_as_double((long long) b);
#else
	double d;
	std::memcpy(&d, &b, 8);
	return d;
#endif
}

// floor(d) and its value as an int, for 0 <= d < 2^31 (true when the
// result is false: the caller then uses the FP64 instructions).  +0.0 and
// every d in [0, 1) give +0.0 and 0.
CPIC_HD bool floor_nonneg(double d, double &f, int &i)
{
	const uint64_t b = to_bits(d);
	if(b >> 63)
		return false;                       // negative (or -0.0): not handled
	const int e = (int) ((b >> 52) & 0x7ff) - 1023;
	if(e < 0)
	{
		f = 0.0;
		i = 0;
		return true;
	}
	if(e > 30)
		return false;                       // >= 2^31, or Inf / NaN
	const uint64_t m = (b & 0xfffffffffffffull) | (1ull << 52);
	const int sh = 52 - e;                  // 22 .. 52 fractional bits
	f = from_bits(b & ~((1ull << sh) - 1ull));
	i = (int) (m >> sh);
	return true;
}

// The compares of the periodic wrap and of the velocity check, from the
// bits (positive doubles order like their bit patterns read as integers).
// Each gives the IEEE compare's result for every finite or infinite d; for a
// NaN d the caller's result is NaN either way and is reported as such.

// d >= L, for a finite L > 0
CPIC_HD bool ge_pos(double d, double L)
{
	return (int64_t) to_bits(d) >= (int64_t) to_bits(L);
}

// d < 0.0 (false for -0.0)
CPIC_HD bool lt_zero(double d)
{
	const int64_t b = (int64_t) to_bits(d);
	return b < 0 && b != INT64_MIN;
}

// |d| > u, for a finite u >= 0 (false for a NaN d, as the IEEE compare)
CPIC_HD bool abs_gt(double d, double u)
{
	const uint64_t a = to_bits(d) & 0x7fffffffffffffffull;
	return a > to_bits(u) && a <= 0x7ff0000000000000ull;
}

// d is +0.0 or -0.0
CPIC_HD bool is_zero(double d)
{
	return (to_bits(d) << 1) == 0;
}

// d is neither infinite nor NaN
CPIC_HD bool is_finite(double d)
{
	return (to_bits(d) & 0x7ff0000000000000ull) != 0x7ff0000000000000ull;
}

// a / d for a finite d and its rounded reciprocal r = rn(1 / d), by
// Markstein's method (IBM J. Res. Dev. 34, 1990): the quotient estimate a r
// corrected once by its exact remainder, which gives the correctly rounded
// quotient for every normal result.  Three fused or plain FP64
// instructions for a division by a constant.  An infinite or NaN estimate is
// returned as it is, as a / d would be.
CPIC_HD double div_by(double a, double d, double r)
{
#ifdef __CUDA_ARCH__
	const double q = __dmul_rn(a, r);
	const double c = __fma_rn(__fma_rn(-q, d, a), r, q);
#else
	const double q = a * r;
	const double c = std::fma(std::fma(-q, d, a), r, q);
#endif
	return is_finite(q) ? c : q;
}

// Division of a tile index by the number of tiles per row without a divide
// instruction: q = t / n = (t * mul) >> sh (a 32 x 32 -> 64-bit product and
// a shift), exact for every t < 2^30 and n in [1, 2^30).  With D = 2n,
// c = ceil(log2 D) and mul = ceil(2^(31+c) / D) < 2^32: t * mul / 2^(30+c)
// = 2t * mul / 2^(31+c) = t/n + 2t e / (D 2^(31+c)) with e = mul D -
// 2^(31+c) < D <= 2^c, an excess below 1/n for 2t < 2^31.  For a power of
// two n, mul = 2^31 and the result is t >> log2 n.
CPIC_HD void div_init(uint32_t n, uint32_t &mul, int &sh)
{
	const uint64_t D = 2ull * n;
	int c = 0;
	while((1ull << c) < D)
		c++;
	mul = (uint32_t) (((1ull << (31 + c)) + D - 1) / D);
	sh = 30 + c;
}

CPIC_HD uint32_t div_q(uint32_t t, uint32_t mul, int sh)
{
	return (uint32_t) (((uint64_t) t * mul) >> sh);
}

// mag / 2^k rounded to the nearest integer, ties to even, for k >= 0.
CPIC_HD uint64_t rshift_rne(uint64_t mag, int k)
{
	if(k == 0)
		return mag;
	if(k > 64)
		return 0;                           // mag < 2^64 <= half of 2^k
	const uint64_t q = k == 64 ? 0 : mag >> k;
	const uint64_t r = k == 64 ? mag : mag & ((1ull << k) - 1ull);
	const uint64_t half = 1ull << (k - 1);
	return q + ((r > half || (r == half && (q & 1ull))) ? 1ull : 0ull);
}

// hi = rn(v), lo = rn((v - hi) * 2^lo_exp) for a finite v with |v| < 2^62
// (false otherwise: the caller then uses the FP64 instructions); rn rounds
// to the nearest integer, ties to even, as __double2ll_rn does.  v - hi is
// exact in FP64 and so is its product by a power of two, so lo's only
// rounding is the final one, which this reproduces on the integer
// fraction.
CPIC_HD bool split_fixed(double v, int lo_exp, long long &hi, long long &lo)
{
	const uint64_t b = to_bits(v);
	const bool neg = (b >> 63) != 0;
	const int E = (int) ((b >> 52) & 0x7ff);
	if(E == 0x7ff)
		return false;                       // Inf / NaN
	if(E == 0)
	{
		if((b & 0xfffffffffffffull) != 0)
			return false;                       // subnormal: not handled
		hi = 0;
		lo = 0;
		return true;
	}
	const int e = E - 1023;
	if(e >= 62)
		return false;
	const uint64_t m = (b & 0xfffffffffffffull) | (1ull << 52);
	const int sh = 52 - e;                  // fractional bits of |v| = m 2^-sh
	uint64_t him, lom;
	if(sh <= 0)
	{
		him = m << (-sh);                       // an integer: nothing below
		lom = 0;
		hi = neg ? -(long long) him : (long long) him;
		lo = 0;
		return true;
	}
	// |v| = m 2^-sh; its integer part q, remainder r < 2^sh (sh up to 1074:
	// beyond 63 fractional bits q is 0 and r is m itself)
	const uint64_t q = sh >= 64 ? 0 : m >> sh;
	const bool r_all = sh >= 64;
	const uint64_t r = r_all ? m : m & ((1ull << sh) - 1ull);
	// round half to even: up when r > 2^(sh-1), or equal and q odd
	bool up;
	if(sh > 64)
		up = false;                             // r = m < 2^53 < 2^(sh-1)
	else
	{
		const uint64_t half = 1ull << (sh - 1);
		up = r > half || (r == half && (q & 1ull));
	}
	him = q + (up ? 1ull : 0ull);
	// |v| - him = f 2^-sh, f = r - up 2^sh (signed; |f| <= 2^(sh-1));
	// lo = rn(f 2^(lo_exp - sh)), symmetric in the sign of f
	bool fneg;
	uint64_t fmag;
	if(!up)
	{
		fneg = false;
		fmag = r;
	}
	else
	{
		fneg = true;                            // r - 2^sh < 0 (sh <= 64 here)
		fmag = sh == 64 ? (uint64_t) 0 - r : (1ull << sh) - r;
	}
	const int k = sh - lo_exp;              // right shift of the fraction
	if(k <= 0)
	{
		if(-k >= 64 || (fmag >> (63 + k)) != 0)
			return false;                       // would not fit in 63 bits
		lom = fmag << (-k);
	}
	else
		lom = rshift_rne(fmag, k);
	const bool lneg = neg != fneg;
	hi = neg ? -(long long) him : (long long) him;
	lo = lneg ? -(long long) lom : (long long) lom;
	return true;
}

// ------------------------------------------------------------------------
// FP64 arithmetic on the integer pipe.
//
// A positive normal double as its significand and exponent: (h:l) 2^(e - 63)
// with bit 63 of the 64-bit h:l set and its low 11 bits zero.  The
// operations below are IEEE 754's, rounded to nearest even, worked out on
// these integers: the exact product or difference, then one rounding to 53
// bits.  A product takes four 32 x 32 -> 64-bit multiplies and about 20
// other instructions (7 clocks of an SM per warp), an FP64 multiply 20
// clocks of its own pipe, which stays free for the rest of the particle's
// arithmetic.  Operands that are zero, subnormal, negative or not finite are
// not handled (false): the caller then uses the FP64 instructions.
struct Pos {
	uint32_t h, l;
	int e;
};

CPIC_HD bool pos_of(double d, Pos &p)
{
	const uint64_t b = to_bits(d);
	const uint32_t f = (uint32_t) (b >> 52);        // sign and exponent
	p.h = (uint32_t) (b >> 21) | 0x80000000u;
	p.l = (uint32_t) b << 11;
	p.e = (int) f - 1023;
	return f - 1u < 2046u;                  // positive, normal, finite
}

CPIC_HD uint64_t pos_bits(Pos p) { return (uint64_t) p.h << 32 | p.l; }

// The double of p; its exponent must be that of a normal double (pos_normal).
CPIC_HD double pos_val(Pos p)
{
	return from_bits((pos_bits(p) >> 11) + ((uint64_t) (uint32_t) (p.e + 1022) << 52));
}

CPIC_HD bool pos_normal(Pos p)
{
	return (uint32_t) (p.e + 1022) < 2046u;
}

// The upper word of (hi:lo) << n, n < 32.
CPIC_HD uint32_t funnel_l(uint32_t lo, uint32_t hi, int n)
{
#ifdef __CUDA_ARCH__
	return __funnelshift_l(lo, hi, n);
#else
	return n ? hi << n | lo >> (32 - n) : hi;
#endif
}

CPIC_HD int clz32(uint32_t v)
{
#ifdef __CUDA_ARCH__
	return __clz((int) v);
#else
	return v ? __builtin_clz(v) : 32;
#endif
}

CPIC_HD int clz64(uint64_t v)
{
#ifdef __CUDA_ARCH__
	return __clzll((long long) v);
#else
	return v ? __builtin_clzll(v) : 64;
#endif
}

// h:l (bit 63 set), the bits below it by whether any is set, rounded to 53
// bits: times 2^(e - 63).  The sum's bit 63 is clear only when it wrapped,
// i.e. rounded up to the next power of two.
CPIC_HD Pos pos_round(uint32_t h, uint32_t l, uint32_t below, int e)
{
	l |= below < 1u ? below : 1u;
	const uint64_t t = ((uint64_t) h << 32 | l) + (0x3ffu + ((l >> 11) & 1u));
	const uint32_t th = (uint32_t) (t >> 32);
	Pos r;
	r.h = th | 0x80000000u;
	r.l = (uint32_t) t & ~0x7ffu;
	r.e = e + 1 - (int) (th >> 31);
	return r;
}

// The 128-bit product h:l1:l0 (h >= 2^62 as 64 bits) times 2^(e - 127),
// rounded to 53 bits.
CPIC_HD Pos pos_norm(uint64_t h, uint32_t l1, uint32_t l0, int e)
{
	const uint32_t hh = (uint32_t) (h >> 32), hl = (uint32_t) h;
	const int n = (int) (hh >> 31) ^ 1;     // shift by one, or not
	return pos_round(funnel_l(hl, hh, n), funnel_l(l1, hl, n), l1 << n | l0, e - n);
}

// rn(a b)
CPIC_HD Pos pos_mul(Pos a, Pos b)
{
	const uint64_t p = (uint64_t) a.l * b.l;
	const uint64_t t = (uint64_t) a.l * b.h + (uint32_t) (p >> 32);
	const uint64_t u = (uint64_t) a.h * b.l + (uint32_t) t;
	const uint64_t h = (uint64_t) a.h * b.h + (uint32_t) (t >> 32) + (uint32_t) (u >> 32);
	return pos_norm(h, (uint32_t) u, (uint32_t) p, a.e + b.e + 1);
}

// rn(i b) for an integer i >= 1
CPIC_HD Pos pos_mul_int(uint32_t i, Pos b)
{
	const int c = clz32(i);
	const uint32_t a = i << c;
	const uint64_t u = (uint64_t) a * b.l;
	const uint64_t h = (uint64_t) a * b.h + (uint32_t) (u >> 32);
	return pos_norm(h, (uint32_t) u, 0u, 32 - c + b.e);
}

// v << n and v >> n for 0 <= n < 64 (n is reduced to that where a result is
// not used).
CPIC_HD uint64_t shl64(uint64_t v, int n) { return v << (n & 63); }
CPIC_HD uint64_t shr64(uint64_t v, int n) { return v >> (n & 63); }

// The functions below have no branches where the lanes of a warp would take
// both sides anyway; where the returned flag is false the other results are
// meaningless.

// rn(1 - a) for 0 < a < 1 (a.e < 0)
CPIC_HD Pos pos_one_minus(Pos a)
{
	// in units of 2^-64: x = 2^64 - floor(a 2^64), less one (an odd number,
	// never a tie) when a bit of a lies below the units.  a >= 1/2 leaves an
	// exact difference with leading zeros, a < 1/2 a full word to be rounded
	// to a multiple of 2^11.
	const int sh = -1 - a.e;                // 0 ...
	const uint64_t am = pos_bits(a);
	const bool far = sh >= 64;
	const uint64_t q = far ? 0ull : shr64(am, sh);
	const bool rest = far || shl64(q, sh) != am;
	const uint64_t x = 0ull - (q | (rest ? 1ull : 0ull));
	const int c = clz64(x);
	const uint64_t m = shl64(x, c);
	return pos_round((uint32_t) (m >> 32), (uint32_t) m, 0u, -1 - c);
}

// The cell index and the offset in the cell of position x > 0, as the FP64
// sequence  i0 = floor(x idx);  rel = (x - i0 dx) idx  gives them; false
// where a step is not handled (i0 out of range, an offset that is zero,
// negative or 1 or more, a difference that would have to be rounded).
CPIC_HD bool pos_rel(Pos x, Pos dx, Pos idx, int &i0, Pos &rel)
{
	const Pos p = pos_mul(x, idx);
	if(p.e > 30)
		return false;
	uint32_t i = 0;
	Pos d = x;                              // x - 0 dx
	// (a branch: the first cell is rare, and selecting between its offset
	// and the others' took 3 % of the FP64 form's particle kernel)
	if(p.e >= 0)
	{
		i = p.h >> (31 - p.e);
		const Pos s = pos_mul_int(i, dx);
		const int k = x.e - s.e;
		// x is within a factor two of i dx: the difference is exact, in units
		// of the smaller one's last place
		const int kx = k > 0 ? 10 : 11, ks = k < 0 ? 10 : 11;
		const int64_t v = (int64_t) (pos_bits(x) >> kx) - (int64_t) (pos_bits(s) >> ks);
		if((unsigned) (k + 1) > 2u || v <= 0 || (v >> 53) != 0)
			return false;
		const int c = clz64((uint64_t) v);
		const uint64_t m = shl64((uint64_t) v, c);
		d.h = (uint32_t) (m >> 32);
		d.l = (uint32_t) m;
		d.e = (k > 0 ? s.e : x.e) + 11 - c;
	}
	i0 = (int) i;
	rel = pos_mul(d, idx);
	return rel.e < 0;
}

// hi = rn(v), lo = rn((v - hi) 2^lo_exp), both negated when neg, as
// split_fixed, for 1 <= v < 2^62 and 1 <= lo_exp <= 63 (false otherwise).
CPIC_HD bool pos_split(Pos v, bool neg, int lo_exp, long long &hi, long long &lo)
{
	const int sh = 63 - v.e;                // 2 .. 63 fractional bits of m
	const uint64_t m = pos_bits(v);
	const uint64_t q = shr64(m, sh);
	const uint64_t r = shl64(m, 64 - sh);   // the fraction, in units of 2^-64
	// up past one half, or at it from an odd integer
	const bool up = r > (1ull << 63) - (q & 1ull);
	const uint64_t f = up ? 0ull - r : r;   // |v - hi|
	const uint64_t g = shr64(f, 64 - lo_exp);
	const uint64_t rem = shl64(f, lo_exp);
	const bool up2 = rem > (1ull << 63) - (g & 1ull);
	const uint64_t h = q + (up ? 1ull : 0ull), l = g + (up2 ? 1ull : 0ull);
	hi = neg ? -(long long) h : (long long) h;
	lo = neg != up ? -(long long) l : (long long) l;
	return (unsigned) v.e < 62u;
}

// The cell index and the offset in the cell of position x > 0 from the exact
// product x idx: i0 = floor(x idx), f = rn(x idx - i0), as one fused
// multiply-add gives it; false where i0 is out of range or f is 0 or rounds to
// 1.
CPIC_HD bool pos_frac(Pos x, Pos idx, int &i0, Pos &f)
{
	const uint64_t p = (uint64_t) x.l * idx.l;
	const uint64_t t = (uint64_t) x.l * idx.h + (uint32_t) (p >> 32);
	const uint64_t u = (uint64_t) x.h * idx.l + (uint32_t) t;
	const uint64_t h = (uint64_t) x.h * idx.h + (uint32_t) (t >> 32) + (uint32_t) (u >> 32);
	const uint64_t l = u << 32 | (uint32_t) p;
	// the product is (h:l) 2^(e - 127): e + 1 integer bits
	const int ib = x.e + idx.e + 2;
	const bool some = ib > 0;
	const int n = some ? ib : 0;
	i0 = some ? (int) ((uint32_t) (h >> 32) >> ((32 - n) & 31)) : 0;
	const uint64_t fh = shl64(h, n) | (some ? shr64(l, 64 - n) : 0ull);
	const uint64_t fl = shl64(l, n);
	const int c = clz64(fh);
	const uint64_t m = shl64(fh, c) | (c ? shr64(fl, 64 - c) : 0ull);
	const uint64_t below = shl64(fl, c);
	f = pos_round((uint32_t) (m >> 32), (uint32_t) m, (uint32_t) (below >> 32) | (uint32_t) below,
			(some ? -1 : ib - 1) - c);
	return (ib <= 31) & (fh != 0) & (f.e < 0);
}

// A positive normal float (24 bits: l is 0).
CPIC_HD bool pos_of(float a, Pos &p)
{
#ifdef __CUDA_ARCH__
	const uint32_t b = __float_as_uint(a);
#else
	uint32_t b;
	std::memcpy(&b, &a, 4);
#endif
	const uint32_t f = b >> 23;
	p.h = b << 8 | 0x80000000u;
	p.l = 0;
	p.e = (int) f - 127;
	return f - 1u < 254u;
}

// rn(a b) for a of 24 bits (a.l == 0)
CPIC_HD Pos pos_mul24(Pos a, Pos b)
{
	const uint64_t u = (uint64_t) a.h * b.l;
	const uint64_t h = (uint64_t) a.h * b.h + (uint32_t) (u >> 32);
	return pos_norm(h, (uint32_t) u, 0u, a.e + b.e + 1);
}

// a b for a and b of 24 bits: exact in 48
CPIC_HD Pos pos_mul24x24(Pos a, Pos b)
{
	const uint64_t h = (uint64_t) a.h * b.h;
	const int n = (int) (h >> 63) ^ 1;
	Pos r;
	r.h = (uint32_t) ((h << n) >> 32);
	r.l = (uint32_t) (h << n);
	r.e = a.e + b.e + 1 - n;
	return r;
}

// v rounded to the nearest integer, ties to even, negated when neg; false for
// v >= 2^62.
CPIC_HD bool pos_rint(Pos v, bool neg, long long &out)
{
	const int sh = 63 - v.e;                // 2 .. 64 fractional bits where v >= 1/2
	const uint64_t m = pos_bits(v);
	const bool none = v.e < 0;              // no integer bits
	const uint64_t q0 = none ? 0ull : shr64(m, sh);
	const uint64_t r = none ? (v.e == -1 ? m : 0ull) : shl64(m, 64 - sh);
	const uint64_t q = q0 + (r > (1ull << 63) - (q0 & 1ull) ? 1ull : 0ull);
	out = neg ? -(long long) q : (long long) q;
	return v.e < 62;
}

} // namespace bits
} // namespace cpic
