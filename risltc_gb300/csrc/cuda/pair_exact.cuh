// pair_exact.cuh - exact numerics on Blackwell's paired FP32 instructions
// (FADD2 / FFMA2 on float2): two independent scalar computations in the two
// lanes, each operation rounded as its scalar counterpart.
//
// A paired multiply and a paired add that consumes it must not become one
// fused operation, and the code generator fuses them (also with
// --fmad=false, and also when the product is written as fma(a, b, -0) with a
// literal -0: measured, every exact frame then differed from the oracle).  So
// the product is a fused multiply-add whose addend is a -0 that only the host
// knows (a kernel parameter): RN(a * b + -0) is RN(a * b) for every a and b,
// signs of zeros included, and nothing may be folded into it.
//
// A paired instruction occupies the FMA pipe for two issue cycles (measured:
// 59 paired against 115 scalar thread instructions per clock and SM), so the
// gain is in issue slots, which scalar exact numerics runs out of first.
#pragma once
#include "shade_device.cuh"

namespace risltc {

RL_DEV float2 pair(float a) { return make_float2(a, a); }

struct PairExact {
	float2 neg_zero;
	RL_DEV float2 mul(float2 a, float2 b) const { return __ffma2_rn(a, b, neg_zero); }
	static RL_DEV float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }
	// a - b: b * -1 is exact.
	static RL_DEV float2 sub(float2 a, float2 b) { return __ffma2_rn(b, pair(-1.0f), a); }
	static RL_DEV float2 fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
};

RL_DEV float rsqrt_approx(float x) {
	float y;
	asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
	return y;
}

// RN(sqrt(d)) in both lanes, for every finite d of 2^-76 or more (as words
// [kRootMin, kRootMax]), where y is the approximate reciprocal root: one Newton
// step from g = RN(d y), g + (d - g^2) y / 2, with the remainder and the sum
// each in one fused multiply-add.
//
// Why it rounds correctly (the argument of Cornea-Hasegan, Golliver and
// Markstein, "Correctness proofs outline for Newton-Raphson based
// floating-point divide and square root algorithms", ARITH-14, 1999): let
// y = (1 + e) / sqrt(d) with |e| <= 2^-22.9 (the documented error of
// rsqrt.approx), g = (1 + t) sqrt(d) with |t| <= 2^-22.3 and E the remainder's
// rounding, |E| <= 2^-24.  Before its own rounding the sum is
// sqrt(d) (1 + t - (1 + e)(1 + E)(t + t^2 / 2)), off from sqrt(d) by less than
// t^2 / 2 + |t e| + |t E| < 2^-43 of it.  It can be rounded to the wrong side
// only where a midpoint M of two neighbouring floats lies as close to sqrt(d).
// In units where these floats are the integers of [2^23, 2^24), M = k + 1/2 and
// d is a multiple of 2^23, so d - M^2 is never 0 and M is that close only if
// k^2 + k lies within 64 of a multiple of 2^23: two k in 2^23 per even residue,
// of the order of a hundred significands.  They depend on d's significand and
// the parity of its exponent alone, as every step here does while the
// remainder, a multiple of 2^-46 d, is a normal number: d >= 2^-76.  A GPU test
// compares the root with __fsqrt_rn on every float of the range, these
// significands among them.  (Where the remainder loses bits it does go wrong:
// on 1,831,424 of the normal floats up to 2^-102, and on none above.)
constexpr uint32_t kRootMin = 0x19800000u, kRootMax = 0x7f7fffffu;
RL_DEV float2 root_from_rsqrt(const PairExact& o, float2 d, float2 y) {
	const float2 g = o.mul(d, y);
	// y / 2: y is normal, so its exponent field drops by one.
	const float2 h = make_float2(__int_as_float(__float_as_int(y.x) - 0x00800000),
	                             __int_as_float(__float_as_int(y.y) - 0x00800000));
	return o.fma(o.fma(make_float2(-g.x, -g.y), g, d), h, g);
}

// -RN(1 / RN(sqrt(d))) in both lanes over the same range: the reciprocal is
// Markstein's correction of the hardware's (IBM J. Res. Dev. 34(1), 1990),
// taken of -s so that no sign has to change.  Ten operations against fourteen
// of rcp_markstein(sqrt_tuckerman(d)), none of them a comparison.  A GPU test
// compares both lanes with __frcp_rn(__fsqrt_rn(d)) on every float of the
// range.
RL_DEV float2 rsqrt_negated(const PairExact& o, float2 d) {
	const float2 s = root_from_rsqrt(o, d, make_float2(rsqrt_approx(d.x), rsqrt_approx(d.y)));
	const float2 nr = make_float2(rcp_approx(-s.x), rcp_approx(-s.y));
	return o.fma(nr, o.fma(s, nr, pair(1.0f)), nr);
}

// The negated rational fit of integrate_edge, -RN(a(x) / b(x)), in both lanes
// for x in (0, 1 + 2^-15] (the cosine of two normalised vectors less than 90
// degrees apart): Markstein's quotient, one residual correction of a * rcp(b)
// (IBM J. Res. Dev. 34(1), 1990), here from the uncorrected reciprocal and
// taken of -b.  That theorem wants the reciprocal correctly rounded, so what
// stands for this form is the test of all its inputs: x is the only one.  A GPU
// test compares it with __fdiv_rn(a(x), b(x)) on every float of the range.
RL_DEV float2 edge_fit_negated(const PairExact& o, float2 x) {
	const float2 a = o.add(pair(0.8543985f), o.mul(o.add(pair(0.4965155f), o.mul(pair(0.0145206f), x)), x));
	const float2 b = o.add(pair(3.4175940f), o.mul(o.add(pair(4.1616724f), x), x));
	const float2 nz = make_float2(rcp_approx(-b.x), rcp_approx(-b.y));
	const float2 nq = o.mul(a, nz);
	return o.fma(o.fma(b, nq, a), nz, nq);
}

}  // namespace risltc
