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

// -RN(1 / RN(sqrt(d))) in both lanes, for every finite d of 2^-76 or more
// (as words [kRootMin, kRootMax]).  The root is g = d * rsqrt(d) corrected once: the
// remainder d - g^2 comes from one fused multiply-add and is added with half
// the approximate reciprocal root; the reciprocal is Markstein's correction
// of the hardware reciprocal, taken of -s so that no sign has to change.
// Ten operations against fourteen of rcp_markstein(sqrt_tuckerman(d)), none
// of them a comparison.  A GPU test compares both lanes with
// __frcp_rn(__fsqrt_rn(d)) on every float of the range.
constexpr uint32_t kRootMin = 0x19800000u, kRootMax = 0x7f7fffffu;
RL_DEV float2 rsqrt_negated(const PairExact& o, float2 d) {
	const float2 y = make_float2(rsqrt_approx(d.x), rsqrt_approx(d.y));
	const float2 g = o.mul(d, y);
	// y / 2: y is normal, so its exponent field drops by one.
	const float2 h = make_float2(__int_as_float(__float_as_int(y.x) - 0x00800000),
	                             __int_as_float(__float_as_int(y.y) - 0x00800000));
	const float2 s = o.fma(o.fma(make_float2(-g.x, -g.y), g, d), h, g);
	const float2 nr = make_float2(rcp_approx(-s.x), rcp_approx(-s.y));
	return o.fma(nr, o.fma(s, nr, pair(1.0f)), nr);
}

// The negated rational fit of integrate_edge, -RN(a(x) / b(x)), in both lanes
// for x in (0, 1 + 2^-15] (the cosine of two normalised vectors less than 90
// degrees apart): one residual correction of a * rcp(b), taken of -b.  A GPU
// test compares it with __fdiv_rn(a(x), b(x)) on every float of the range.
RL_DEV float2 edge_fit_negated(const PairExact& o, float2 x) {
	const float2 a = o.add(pair(0.8543985f), o.mul(o.add(pair(0.4965155f), o.mul(pair(0.0145206f), x)), x));
	const float2 b = o.add(pair(3.4175940f), o.mul(o.add(pair(4.1616724f), x), x));
	const float2 nz = make_float2(rcp_approx(-b.x), rcp_approx(-b.y));
	const float2 nq = o.mul(a, nz);
	return o.fma(o.fma(b, nq, a), nz, nq);
}

}  // namespace risltc
