// Double-precision operations on the integer pipes, correctly rounded (the bits of the FP64 unit).
//
// GB300 issues 2 FP64 lane-operations per SM and clock, one warp instruction per 64 clocks of a
// scheduler, and the integrators saturate that pipe while the scheduler's other 60 issue slots pass
// unused.  Logic, shifts, selects and comparisons issue at 64 lanes per SM and clock, IMAD at 64
// beside them (a pipe of its own), 32-bit additions, minima and maxima at 128 (measured).  A double
// addition written for these pipes takes 75 clocks of a scheduler against the FP64 pipe's 64, and
// the two overlap: a DFMA beside it adds 6 clocks.  Sharing a sub-step's operations between the
// pipes is therefore worth almost a second FP64 unit.
//
// The results are IEEE 754 round-to-nearest-even, bit for bit, so the CPU oracle replays the same
// operations whichever pipe they ran on.  Operands for which the integer form does not hold (a sum
// of zero or cancelled below the top 32 bits, magnitudes 2^32 apart, exponents near the ends of the
// range, infinities and NaN) set a flag instead; the caller checks the flags of a batch of operations
// with one vote and, where any lane has one set, redoes the batch on the FP64 pipe.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "nlc_device.cuh"
#include "nlc_internal.h"

namespace nlc {

// What a batch of integer-pipe operations saw, as extremes (minima and maxima issue at twice the
// rate of predicates): the batch is invalid when an exponent difference, an exponent or the high
// word of a sum was out of the form's range.
struct IntFlags {
	uint32_t dmax = 0;    // largest exponent difference: up to 31
	uint32_t exmax = 0;   // largest (biased exponent - 64), mod 2^32: up to 1976
	int32_t rmin = 1;     // smallest high word of a sum, or alignment of a square: from 1
	__device__ __forceinline__ bool bad() const { return (dmax > 31u) | (exmax > 1976u) | (rmin <= 0); }
};

// Whether a lane that is here now has to redo its operations on the FP64 pipe.  The vote keeps the warp
// together: a lane that branched off alone can run what follows apart from the others, every FP64
// instruction of it twice.  Where the operations to redo are few (up to about eight), they belong in a
// function that is not inlined: under a branch they become predicated instructions, which occupy the
// pipe whether redone or not.
__device__ __forceinline__ bool any_bad(const IntFlags &f) { return __any_sync(__activemask(), f.bad()); }

__device__ __forceinline__ uint64_t mul_wide(uint32_t a, uint32_t b) {
	uint64_t r;
	asm("mul.wide.u32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
	return r;
}
__device__ __forceinline__ uint64_t mad_wide(uint32_t a, uint32_t b, uint64_t c) {
	uint64_t r;
	asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
	return r;
}
__device__ __forceinline__ uint32_t lo32(uint64_t a) { return uint32_t(a); }
__device__ __forceinline__ uint32_t hi32(uint64_t a) { return uint32_t(a >> 32); }

// a + b, the high word of b given apart (int_sub flips its sign).  Both significands are placed with the leading bit at bit 61 of 64 (carry at 62, sign at
// 63), 9 bits below the last one kept; the smaller operand is shifted right, its lost bits ORed
// into its lowest one, and added or (two's complement) subtracted; the sum's leading bit goes to
// bit 62 and the 10 bits below the 53 kept are rounded off.  The hidden bit is added into the
// exponent field, which also takes the carry of the rounding.
__device__ __forceinline__ double int_add_words(double a, uint32_t bh, uint32_t bl, IntFlags &f) {
	const uint32_t ah = __double2hiint(a), al = __double2loint(a);
	const uint32_t aa = ah & 0x7fffffffu, ba = bh & 0x7fffffffu;
	const bool swap = aa < ba;   // by the high words: equal ones cancel and are flagged where it matters
	const uint32_t xh = swap ? bh : ah, xl = swap ? bl : al, yl = al + bl - xl;
	const uint32_t xa = max(aa, ba), ya = min(aa, ba);
	const uint32_t ex = xa >> 20, d = ex - (ya >> 20);
	const uint32_t neg = uint32_t(int32_t(ah ^ bh) >> 31);   // all ones: magnitudes subtract
	const uint32_t mx = (xa & 0xfffffu) | 0x100000u, my = (ya & 0xfffffu) | 0x100000u;
	const uint32_t xhi = __funnelshift_l(xl, mx, 9), xlo = (xl << 9) - neg;   // the + 1 of the two's complement
	const uint32_t yhi = __funnelshift_l(yl, my, 9), ylo = yl << 9;
	const uint32_t lost = __funnelshift_r(0u, ylo, d);
	const uint32_t slo = (__funnelshift_r(ylo, yhi, d) | min(lost, 1u)) ^ neg, shi = (yhi >> (d & 31u)) ^ neg;
	uint32_t rl, rh;
	asm("{add.cc.u32 %0, %2, %3; addc.u32 %1, %4, %5;}" : "=r"(rl), "=r"(rh) : "r"(xlo), "r"(slo), "r"(xhi), "r"(shi));
	uint32_t lead;   // left shift that brings the leading bit of rh to bit 31
	asm("bfind.shiftamt.u32 %0, %1;" : "=r"(lead) : "r"(rh));
	const uint32_t s = lead - 1u;
	const uint32_t nh = __funnelshift_l(rl, rh, s), nl = rl << (s & 31u);
	const uint32_t half = ((nl >> 10) & 1u) + 0x1ffu;   // to nearest, ties to even
	uint32_t ol, oh;
	asm("{add.cc.u32 %0, %2, %3; addc.u32 %1, %4, 0;}" : "=r"(ol), "=r"(oh) : "r"(nl), "r"(half), "r"(nh));
	f.dmax = max(f.dmax, d);
	f.exmax = max(f.exmax, ex - 64u);
	f.rmin = min(f.rmin, int32_t(rh));
	return __hiloint2double(int(((oh >> 10) + (ex - s) * 0x100000u) | (xh & 0x80000000u)), int(__funnelshift_r(ol, oh, 10)));
}

__device__ __forceinline__ double int_add(double a, double b, IntFlags &f) {
	return int_add_words(a, __double2hiint(b), __double2loint(b), f);
}
__device__ __forceinline__ double int_sub(double a, double b, IntFlags &f) {
	return int_add_words(a, __double2hiint(b) ^ 0x80000000u, __double2loint(b), f);
}

// a b: the exact product of the 53-bit significands, leading bit at 104 or 105 of 128, the low 32 bits
// ORed into the rounding as one.
__device__ __forceinline__ double int_mul(double a, double b, IntFlags &f) {
	const uint32_t ah = __double2hiint(a), a0 = __double2loint(a), bh = __double2hiint(b), b0 = __double2loint(b);
	const uint32_t a1 = (ah & 0xfffffu) | 0x100000u, b1 = (bh & 0xfffffu) | 0x100000u;
	const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
	const uint64_t low = mul_wide(a0, b0);
	const uint64_t mid = mad_wide(a0, b1, mad_wide(a1, b0, uint64_t(hi32(low))));
	const uint64_t top = mad_wide(a1, b1, uint64_t(hi32(mid)));   // the product's bits from 64 on
	const uint32_t carry = hi32(top) >> 9;                        // 1: leading bit at 105
	// the 53 bits kept in (w2, w1), the rest in w0 with its first bit at bit 31
	const uint32_t up = 0x1000u >> carry;
	const uint64_t u0 = mul_wide(lo32(mid), up), u1 = mul_wide(lo32(top), up);
	const uint32_t w0 = lo32(u0) | min(lo32(low), 1u), w1 = lo32(u1) + hi32(u0), w2 = hi32(top) * up + hi32(u1);
	// to nearest, ties to even: up where w0, its lowest bit replaced by w1's at a tie, exceeds 2^31
	const uint32_t inc = (w0 | (w1 & 1u)) > 0x80000000u ? 1u : 0u;
	uint32_t ol, oh;
	asm("{add.cc.u32 %0, %2, %3; addc.u32 %1, %4, 0;}" : "=r"(ol), "=r"(oh) : "r"(w1), "r"(inc), "r"(w2));
	const uint32_t e = ea + eb + carry;   // result exponent + 1023, less the hidden bit's 1 below
	f.exmax = max(max(f.exmax, ea - 64u), max(eb - 64u, e - 1088u));
	return __hiloint2double(int((oh + (e - 1024u) * 0x100000u) ^ ((ah ^ bh) & 0x80000000u)), int(ol));
}

// An addend K > 0 of int_square_plus: its significand with the leading bit at bit 62 of 64, its
// exponent plus 1023, and the exponent field (less the hidden bit) that the result starts from.
__device__ __forceinline__ IntAddend int_addend(double K) {
	const uint32_t h = __double2hiint(K), l = __double2loint(K), m = (h & 0xfffffu) | 0x100000u;
	return {l << 10, __funnelshift_l(l, m, 10), int32_t(h >> 20) + 1023, (h & 0x7ff00000u) - 0x100000u};
}

// c c + K for K of an ordinary positive exponent (the caller's check) and c c below K's next power of
// two (flagged): the exact square of the 64-bit significand, shifted right to K's scale with the lost
// bits ORed into the lowest one (bits of the square below 2^64 exist exactly when the significand's
// low word is not zero), added to K's and rounded at K's exponent or the next.
__device__ __forceinline__ double int_square_plus(double c, const IntAddend &K, IntFlags &f) {
	const uint32_t ch = __double2hiint(c), cl = __double2loint(c);
	const uint32_t mh = __funnelshift_l(cl, ch, 11) | 0x80000000u, ml = cl << 11;
	const int32_t s = K.scale - 2 * int32_t((ch >> 20) & 0x7ffu);
	// floor(m^2 / 2^64) = mh^2 + floor((mh ml + floor(ml^2 / 2^33)) / 2^31)
	const uint64_t cross = mad_wide(mh, ml, uint64_t(hi32(mul_wide(ml, ml)) >> 1));
	const uint64_t sq = mad_wide(mh, mh, cross >> 31);
	uint64_t aligned, lost;
	asm("shr.u64 %0, %1, %2;" : "=l"(aligned) : "l"(sq), "r"(s));        // shifts of 64 and more give 0
	asm("shl.b64 %0, %1, %2;" : "=l"(lost) : "l"(sq), "r"(64 - s));
	const uint32_t sticky = min(lo32(lost) | hi32(lost) | ml, 1u);
	uint32_t rl, rh;
	asm("{add.cc.u32 %0, %2, %3; addc.u32 %1, %4, %5;}"
	    : "=r"(rl), "=r"(rh)
	    : "r"(K.lo), "r"(lo32(aligned) | sticky), "r"(K.hi), "r"(hi32(aligned)));
	const uint32_t carry = rh >> 31;                                     // the sum reached the next power of two
	const uint32_t drop = 10u + carry, half = ((rl >> drop) & 1u) + (0x200u << carry) - 1u;
	uint32_t ol, oh;
	asm("{add.cc.u32 %0, %2, %3; addc.u32 %1, %4, 0;}" : "=r"(ol), "=r"(oh) : "r"(rl), "r"(half), "r"(rh));
	const uint32_t top = oh >> drop;                                     // 0 where the rounding wrapped
	f.rmin = min(f.rmin, min(s, int32_t(top)));
	return __hiloint2double(int(top + K.field + carry * 0x100000u), int(__funnelshift_r(ol, oh, drop)));
}

// n as a double, |n| < 2^24: through its FP32 value, exact, whose exponent and significand are moved to the
// double's places.
__device__ __forceinline__ double int_to_double(int n) {
	const uint32_t b = __float_as_uint(float(n));
	const uint32_t h = ((b & 0x7fffffffu) >> 3) + 0x38000000u;
	return __hiloint2double(int(n ? h | (b & 0x80000000u) : 0u), int(b << 29));
}

// The nearest integer to x inv_l, |x| < 4096 (the caller's flag), as the FP64 pipe's x inv_l + 1.5 2^52
// rounds it: from the top 64 bits of the exact product's 106, flagged where the bits below the half
// are all zeros (a tie) or all ones (what was cut off could carry).
__device__ __forceinline__ int int_exp_index(double x, const ExpConsts &c, IntFlags &f) {
	const uint32_t xh = __double2hiint(x), x0 = __double2loint(x), x1 = (xh & 0xfffffu) | 0x100000u;
	const uint64_t mid = mad_wide(x0, c.inv1, mad_wide(x1, c.inv0, uint64_t(hi32(mul_wide(x0, c.inv0)))));
	const uint64_t top = mad_wide(x1, c.inv1, uint64_t(hi32(mid)));
	const uint64_t p = uint64_t(__funnelshift_l(lo32(mid), lo32(top), 22)) |
	                   uint64_t(__funnelshift_l(lo32(top), hi32(top), 22)) << 32;   // the product's bits from 42 on
	const int s = 1073 - int((xh >> 20) & 0x7ffu);   // the half's place in p
	uint64_t twice, below;
	asm("shr.u64 %0, %1, %2;" : "=l"(twice) : "l"(p), "r"(s));        // shifts of 64 and more give 0
	asm("shl.b64 %0, %1, %2;" : "=l"(below) : "l"(p), "r"(64 - s));
	f.rmin = min(f.rmin, s > 63 ? 1 : int((hi32(below) + 1u) >> 1));
	const int n = int((lo32(twice) + 1u) >> 1), neg = int(xh) >> 31;
	return (n ^ neg) - neg;
}

// 1 + a b, |a b| < 1/2 (flagged): the exact product's top 64 bits shifted to the scale of 2^-62, the rest
// ORed into the lowest one, added to or subtracted from 2^62; the sum's leading bit is at 62 or 61.  The
// product is that of two significands, below 4, times 2^-t: below 1/2 from t = 3 on.  a is of an ordinary
// size (the caller's: a polynomial near 1/2), b any double.
__device__ __forceinline__ double int_one_plus(double a, double b, IntFlags &f) {
	const uint32_t ah = __double2hiint(a), a0 = __double2loint(a), bh = __double2hiint(b), b0 = __double2loint(b);
	const uint32_t a1 = (ah & 0xfffffu) | 0x100000u, b1 = (bh & 0xfffffu) | 0x100000u;
	const uint64_t low = mul_wide(a0, b0);
	const uint64_t mid = mad_wide(a0, b1, mad_wide(a1, b0, uint64_t(hi32(low))));
	const uint64_t top = mad_wide(a1, b1, uint64_t(hi32(mid)));
	const uint64_t p = uint64_t(__funnelshift_l(lo32(mid), lo32(top), 22)) |
	                   uint64_t(__funnelshift_l(lo32(top), hi32(top), 22)) << 32;   // the product's bits from 42 on
	const int t = 2046 - int((ah >> 20) & 0x7ffu) - int((bh >> 20) & 0x7ffu);
	uint64_t aligned, lost;
	asm("shr.u64 %0, %1, %2;" : "=l"(aligned) : "l"(p), "r"(t));   // shifts of 64 and more give 0
	asm("shl.b64 %0, %1, %2;" : "=l"(lost) : "l"(p), "r"(64 - t));
	const uint32_t sticky = min(lo32(lost) | hi32(lost) | (lo32(mid) << 22) | lo32(low), 1u);
	const uint32_t neg = uint32_t(int32_t(ah ^ bh) >> 31);
	uint32_t rl, rh;
	asm("{add.cc.u32 %0, %2, %3; addc.u32 %1, %4, 0x40000000;}"
	    : "=r"(rl), "=r"(rh)
	    : "r"((lo32(aligned) | sticky) ^ neg), "r"(0u - neg), "r"(hi32(aligned) ^ neg));
	const uint32_t z = ~rh >> 30 & 1u;   // 1: below 1
	const uint32_t drop = 10u - z, half = ((rl >> drop) & 1u) + (0x200u >> z) - 1u;
	uint32_t ol, oh;
	asm("{add.cc.u32 %0, %2, %3; addc.u32 %1, %4, 0;}" : "=r"(ol), "=r"(oh) : "r"(rl), "r"(half), "r"(rh));
	f.rmin = min(f.rmin, t - 2);
	return __hiloint2double(int((oh >> drop) + 0x3fe00000u - z * 0x100000u), int(__funnelshift_r(ol, oh, drop)));
}

// exp_scaled (nlc_device.cuh) with the table's index, its value as a double, the polynomial's last product
// and (HALF) the sum before it on the integer pipes: 5 or 4 of its 8 operations stay on the FP64 pipe.
// Flagged where exp_scaled leaves its fast path, and somewhat before.
template <bool HALF>
__device__ __forceinline__ double exp_scaled_mixed(double x, const double *__restrict__ table, const FpOnes &k1,
                                                   const ExpConsts &c, IntFlags &f) {
	f.rmin = min(f.rmin, 0x40b00000 - (__double2hiint(x) & 0x7fffffff));   // |x| < 4096: |n| < 2^24
	const int n = int_exp_index(x, c, f);
	const double nf = int_to_double(n);
	double r = dfma(-nf, c.l1, x);
	r = dfma(-nf, c.l2, r);
	const double h = dfma(r, c.c3, c.c2), q = HALF ? int_one_plus(h, r, f) : dfma(h, r, k1.one);
	const double tj = table[n & (kExpTable - 1)];
	const double v = dfma(tj, int_mul(q, r, f), tj);
	const int k = n >> 11, hi = __double2hiint(v);
	f.exmax = max(f.exmax, uint32_t(((hi >> 20) & 0x7ff) + k - 64));
	return __hiloint2double(hi + k * 0x100000, __double2loint(v));
}

}  // namespace nlc
