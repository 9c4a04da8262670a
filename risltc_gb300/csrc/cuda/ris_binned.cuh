// ris_binned.cuh - the RIS candidate phase as a warp-per-tile kernel with
// work binning.
//
// Each warp owns kPixels consecutive pixels (32, 16 or 8: the tile's pixels
// per warp) and takes their candidates in super-chunks of kSuper, each made
// of chunks of kChunk (the tile's candidates per pixel per chunk; 8 or 4).
// Per chunk the warp
//   1. draws every pixel's candidate lights from that pixel's noise stream
//      (the LCG sequence of shading_pass.frag.glsl:728-736: a light draw, then
//      the reservoir draw, per candidate);
//   2. sorts the chunk's (pixel, candidate) items by the light's vertex count
//      with a counting sort over the warp, so that the lanes of one step
//      mostly evaluate polygons with the same number of vertices;
//   3. evaluates the items with each pixel's LTC frame read from shared
//      memory, both LTC spaces at once in the lanes of paired FP32
//      instructions and without branches; an item whose polygon is partially
//      clipped in either space, or outside that form's range, is deferred to
//      a list that the warp evaluates 32 at a time, so the clipping path runs
//      with full warps.
// A frame's super-chunk is a unit; after up to four units (a window) the
// last deferred items of the window are evaluated and
//   4. each lane replays its pixel's reservoir updates in candidate order
//      (insert_in_reservoir, reservoir.glsl:34-41), unit by unit, drawing the
//      same noise again.
// Every p_hat is computed by the same operations on the same values as in
// ris_candidates_kernel and the reservoir sees them in the same order, so the
// reservoir records are bit-identical.
// Restates upstream risltc routines (GPLv3): see NOTICE.
#pragma once
#include <algorithm>
#include <atomic>
#include <type_traits>
#include "pair_exact.cuh"
#include "ris_kernels.cuh"

namespace risltc {

// Blocks per SM the candidate kernel is compiled for (register budget).
// Exact numerics 6 (80 registers): 8.46 ms per 4-frame 1080p launch with
// 16,384 lights against 8.89 with 5, 9.30 with 4 and 9.05 with 7 (8.33 now).
// Fast numerics 5: 1.71 ms per 2-frame 720p launch with 4,096 lights against
// 1.80 with 4 and 1.81 with 6 (1.67 now).
#ifndef RISLTC_BINNED_MIN_BLOCKS_EXACT
#define RISLTC_BINNED_MIN_BLOCKS_EXACT 6
#endif
#ifndef RISLTC_BINNED_MIN_BLOCKS_FAST
#define RISLTC_BINNED_MIN_BLOCKS_FAST 5
#endif

// A warp's p_hat values, [window unit][candidate][pixel lane], live in its
// slot of RisParams::p_hat_scratch (global memory, L2/L1): keeping them out
// of shared memory leaves room in the SM's combined L1/shared storage for
// the light records the candidates read.  A slot holds 4096 values: four
// 32-pixel super-chunks of 32 candidates in the default tile.
constexpr int kPHatSlot = 4096;
// The candidate kernels run at most this many blocks per SM (their grid is
// one resident wave); the p_hat scratch has a slot per warp of such a grid.
constexpr int kCandidateBlocksPerSm = 8;

// Candidates per pixel per super-chunk (measured best: 32 in exact numerics,
// 16 in fast numerics, where the smaller tile leaves more L1 for the lights).
#ifndef RISLTC_BINNED_SUPER_EXACT
#define RISLTC_BINNED_SUPER_EXACT 32
#endif
template <class P> struct BinnedSuper {
	static constexpr int value = RISLTC_BINNED_SUPER_EXACT;
};
template <> struct BinnedSuper<FastNumerics> {
	static constexpr int value = 16;
};
template <class P> struct BinnedMinBlocks {
	static constexpr int value = RISLTC_BINNED_MIN_BLOCKS_EXACT;
};
template <> struct BinnedMinBlocks<FastNumerics> {
	static constexpr int value = RISLTC_BINNED_MIN_BLOCKS_FAST;
};
// A pixel's LTC frame in 7 16-byte words (an odd number of them, so that the
// 16-byte reads of 8 lanes from different pixels spread over the banks):
// word 0 {diffuse albedo, LTC albedo}, then the world-to-shading and
// world-to-cosine matrices (mat4x3, column-major) element by element in
// pairs {shading, cosine}.
//
// The side flip (shading_pass.frag.glsl:424-428) is left out: it negates the
// y row of both matrices (shading_to_cosine couples y with nothing), which
// changes neither z nor any dot product and negates every edge integral, so
// the integrals' magnitudes, and with them p_hat, are the same bit for bit.
constexpr int kFrameQuads = 7;
constexpr int kBinnedWarps = 4;              // warps per block
constexpr int kBins = kMaxLightVertices - 2; // vertex counts 3..8

template <int kSuper, int kPixels, int kChunk> struct WarpTile {
	static constexpr int kItems = kPixels * kChunk;  // items per warp per chunk
	static constexpr int kDeferred = kItems + 32;     // deferred items pending at most
	static_assert(kItems < 1024, "10-bit bin counters");
	static_assert(kSuper % kChunk == 0 && kPixels * kSuper <= 1024, "super-chunk layout (10-bit slots)");
	float4 frame[kPixels][kFrameQuads];
	// Items as light << 10 | slot, slot = candidate of the super-chunk *
	// kPixels + pixel lane (below 1024; lights below 2^22).
	uint32_t item[kItems];
	uint32_t deferred[kDeferred];
	uint8_t deferred_unit[kDeferred];  // the window unit of each deferred item
	uint32_t deferred_count;
};

RL_DEV void store_frame(float4* f, f3 diffuse_albedo, float ltc_albedo, const mat43& w2s, const mat43& w2c) {
	f[0] = make_float4(diffuse_albedo.x, diffuse_albedo.y, diffuse_albedo.z, ltc_albedo);
#pragma unroll
	for (int c = 0; c != 4; c += 2) {
		const f3 s0 = w2s.c[c], s1 = w2s.c[c + 1], c0 = w2c.c[c], c1 = w2c.c[c + 1];
		float4* const q = f + 1 + 3 * (c / 2);
		q[0] = make_float4(s0.x, c0.x, s0.y, c0.y);
		q[1] = make_float4(s0.z, c0.z, s1.x, c1.x);
		q[2] = make_float4(s1.y, c1.y, s1.z, c1.z);
	}
}
// The frame's matrix of one space (0 shading, 1 cosine).
RL_DEV mat43 load_matrix(const float4* f, int space) {
	float e[12];
#pragma unroll
	for (int k = 0; k != 6; ++k) {
		const float4 q = f[1 + k];
		e[2 * k] = space == 0 ? q.x : q.y;
		e[2 * k + 1] = space == 0 ? q.z : q.w;
	}
	mat43 m;
#pragma unroll
	for (int c = 0; c != 4; ++c) m.c[c] = mk3(e[3 * c], e[3 * c + 1], e[3 * c + 2]);
	return m;
}

// A light vertex (slot j of the record) in local space: mat4x3 * vec4(v, 1).
RL_DEV f3 local_vertex(const mat43& t, const float4* record, uint32_t j) {
	const float4 q = __ldg(record + kRecordVertex + j);
	return mul_point(t, mk3(q.x, q.y, q.z));
}

// The integral calculate_ltc gives over the part of the polygon above the
// horizon (mask: the vertices above z = 0, one bit each, at least one),
// streamed: with all vertices above in the record's order, otherwise with
// the clipped vertices produced one at a time in the order of clip_polygon's
// output slots: the cycle [entry, the run above the horizon, exit] starting
// at its rotation, the run's vertices transformed again from the light
// record.  The same values in the same order as clip_polygon followed by
// calculate_ltc, without a vertex array.  -1 when the polygon clips to
// nothing.  With kChecked, uses the branch-free normalisation and edge
// integral and clears ok where they do not apply.
template <class P, bool kChecked>
RL_DEV float clipped_integral(const mat43& t, const float4* record, uint32_t n, uint32_t mask, bool& ok) {
	const bool whole = mask == (1u << n) - 1u;
	const uint32_t k = __popc(mask);
	uint32_t s = 0, vc = n, j0 = 0;
	f3 entry = splat(0.0f), exit = splat(0.0f);
	if (!whole) {
		s = clip_run_start(n, mask);
		if (s == n) return -1.0f;
		const uint32_t e = clip_wrap(s + k - 1, n);
		vc = k + 2;
		entry = iz0<P>(local_vertex(t, record, clip_wrap(s + n - 1, n)), local_vertex(t, record, s));
		exit = iz0<P>(local_vertex(t, record, e), local_vertex(t, record, clip_wrap(e + 1, n)));
		j0 = clip_wrap(vc - clip_rotation(n, k, s), vc);  // cycle element of slot 0
	}
	f3 first = splat(0.0f), prev = splat(0.0f);
	float r = 0.0f;
#pragma unroll 1
	for (uint32_t slot = 0; slot != vc; ++slot) {
		const uint32_t j = clip_wrap(j0 + slot, vc);
		f3 v = local_vertex(t, record, whole ? slot : clip_wrap(s + (j == 0 ? 0 : j - 1), n));
		if (!whole) v = j == 0 ? entry : (j == k + 1 ? exit : v);
		const f3 cur = kChecked ? normalize_checked<P>(v, ok) : normalize<P>(v);
		if (slot == 0)
			first = cur;
		else
			r += kChecked ? integrate_edge_checked<P>(prev, cur, ok) : integrate_edge<P>(prev, cur);
		prev = cur;
	}
	r += kChecked ? integrate_edge_checked<P>(prev, first, ok) : integrate_edge<P>(prev, first);
	return fabsf(r);
}

// One candidate (ltc_cp_candidate, then p_hat = length(color)) with the
// frame in shared memory, of any polygon.  In each space the vertices above
// the horizon are counted first, so that only the polygon that is kept is
// normalised and integrated.
template <class P, bool kChecked>
RL_DEV bool binned_candidate(const float4* f, const float4* record, float& p_hat) {
	// kChecked: the branch-free forms (normalize_checked,
	// integrate_edge_checked, sqrt_checked); false when any of them does not
	// apply (a squared length outside the square root's range, an edge of 90
	// degrees or more), and the caller takes the general forms.
	bool ok = true;
	const float4 head = __ldg(record);
	const uint32_t n = __float_as_uint(head.w);
	const float4 f0 = f[0];
	float integral[2];
#pragma unroll 1
	for (int s = 0; s != 2; ++s) {
		const mat43 t = load_matrix(f, s);
		uint32_t mask = 0;  // bit j: vertex j above the horizon
#pragma unroll 1
		for (uint32_t j = 0; j != n; ++j) mask |= (local_vertex(t, record, j).z > 0.0f ? 1u : 0u) << j;
		const float r = mask == 0 ? -1.0f : clipped_integral<P, kChecked>(t, record, n, mask, ok);
		if (s == 0)
			integral[0] = r;
		else
			integral[1] = r;
	}
	if (kChecked && !ok) return false;
	const f3 radiance = mk3(head.x, head.y, head.z);
	f3 result = splat(0.0f);
	const f3 diffuse = integral[0] < 0.0f ? splat(0.0f) : mul(scale(mk3(f0.x, f0.y, f0.z), integral[0]), radiance);
	result = add(result, diffuse);
	const f3 ggx = integral[1] < 0.0f ? splat(0.0f) : mul(splat(integral[1] * f0.w), radiance);
	const f3 color = add(result, ggx);
	if (kChecked) {
		p_hat = sqrt_checked<P>(dot(color, color), ok);
		return ok;
	}
	p_hat = P::sqrt(dot(color, color));
	return true;
}

// ---------------------------------------------------------------------------
// The same candidate with both spaces in the two lanes of Blackwell's paired
// FP32 instructions (lane .x the shading space, lane .y the cosine space).
// Both spaces walk the same vertices, so every transform, dot product, scale
// and edge-integral step of the two spaces is one paired instruction.
// Exact numerics takes its operations from pair_exact.cuh: each lane performs
// the scalar version's operations on the same operands in the same order, so
// the values are bit-identical.  Fast numerics allows contraction.
template <class P> RL_DEV float2 mad2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
template <class P> RL_DEV float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
template <class P> RL_DEV float2 pmul(float2 a, float2 b) { return __fmul2_rn(a, b); }

struct f3x2 {
	float2 x, y, z;
};
// mat4x3 * vec4(p, 1) in both lanes: ((c0 p.x + c1 p.y) + c2 p.z) + c3.
struct mat43x2 {
	f3x2 c[4];
};
RL_DEV mat43x2 load_pairs(const float4* f) {
	mat43x2 m;
#pragma unroll
	for (int c = 0; c != 4; c += 2) {
		const float4 a = f[1 + 3 * (c / 2)], b = f[2 + 3 * (c / 2)], d = f[3 + 3 * (c / 2)];
		m.c[c] = {make_float2(a.x, a.y), make_float2(a.z, a.w), make_float2(b.x, b.y)};
		m.c[c + 1] = {make_float2(b.z, b.w), make_float2(d.x, d.y), make_float2(d.z, d.w)};
	}
	return m;
}
template <class P> RL_DEV f3x2 mul_point2(const mat43x2& m, float4 q) {
	const float2 px = pair(q.x), py = pair(q.y), pz = pair(q.z);
	f3x2 r;
	r.x = padd<P>(mad2<P>(m.c[2].x, pz, mad2<P>(m.c[1].x, py, pmul<P>(m.c[0].x, px))), m.c[3].x);
	r.y = padd<P>(mad2<P>(m.c[2].y, pz, mad2<P>(m.c[1].y, py, pmul<P>(m.c[0].y, px))), m.c[3].y);
	r.z = padd<P>(mad2<P>(m.c[2].z, pz, mad2<P>(m.c[1].z, py, pmul<P>(m.c[0].z, px))), m.c[3].z);
	return r;
}
template <class P> RL_DEV float2 dot2(const f3x2& a, const f3x2& b) {
	return mad2<P>(a.z, b.z, mad2<P>(a.y, b.y, pmul<P>(a.x, b.x)));
}
template <class P> RL_DEV f3x2 normalize2(const f3x2& a) {
	const float2 d = dot2<P>(a, a);
	const float2 s = make_float2(P::rsqrt(d.x), P::rsqrt(d.y));
	return {pmul<P>(a.x, s), pmul<P>(a.y, s), pmul<P>(a.z, s)};
}
// integrate_edge on both lanes.
template <class P> RL_DEV float2 integrate_edge2(const f3x2& v1, const f3x2& v2) {
	const float2 x = dot2<P>(v1, v2);
	const float2 y = make_float2(fabsf(x.x), fabsf(x.y));
	const float2 a = padd<P>(pair(0.8543985f), pmul<P>(mad2<P>(pair(0.0145206f), y, pair(0.4965155f)), y));
	const float2 b = padd<P>(pair(3.4175940f), pmul<P>(padd<P>(pair(4.1616724f), y), y));
	float2 ts = make_float2(P::div_edge(a.x, b.x), P::div_edge(a.y, b.y));
	if (!(x.x > 0.0f)) ts.x = 0.5f * P::rsqrt(fmax_glsl(1.0f - x.x * x.x, 1e-7f)) - ts.x;
	if (!(x.y > 0.0f)) ts.y = 0.5f * P::rsqrt(fmax_glsl(1.0f - x.y * x.y, 1e-7f)) - ts.y;
	const float2 cz = padd<P>(pmul<P>(v1.x, v2.y), pmul<P>(make_float2(-v1.y.x, -v1.y.y), v2.x));
	return pmul<P>(cz, ts);
}

template <class P>
RL_DEV void binned_candidate_pair(const float4* f, const float4* record, float& p_hat) {
	const float4 head = __ldg(record);
	const uint32_t n = __float_as_uint(head.w);
	const float4 f0 = f[0];
	const mat43x2 t = load_pairs(f);
	// Vertices 0 and 1 first; then iteration j normalises vertex j + 1 while
	// it integrates edge (j - 1, j), so the two dependency chains overlap.
	// The edges are added in calculate_ltc's order: (0, 1), ..., (n - 2,
	// n - 1), then (n - 1, 0).
	const float4 q0 = __ldg(record + kRecordVertex), q1 = __ldg(record + kRecordVertex + 1);
	float4 q = __ldg(record + kRecordVertex + 2);
	f3x2 v = mul_point2<P>(t, q0);
	uint32_t above_s = v.z.x > 0.0f ? 1u : 0u, above_c = v.z.y > 0.0f ? 1u : 0u;  // bit j: vertex j above
	const f3x2 first = normalize2<P>(v);
	v = mul_point2<P>(t, q1);
	above_s |= (v.z.x > 0.0f ? 1u : 0u) << 1;
	above_c |= (v.z.y > 0.0f ? 1u : 0u) << 1;
	f3x2 prev = first, cur = normalize2<P>(v);
	float2 r = pair(0.0f);
#pragma unroll 1
	for (uint32_t j = 1; j != n; ++j) {
		f3x2 next = first;
		if (j + 1 != n) {
			v = mul_point2<P>(t, q);
			q = __ldg(record + kRecordVertex + min(j + 2, (uint32_t) kMaxLightVertices - 1));
			above_s |= (v.z.x > 0.0f ? 1u : 0u) << (j + 1);
			above_c |= (v.z.y > 0.0f ? 1u : 0u) << (j + 1);
			next = normalize2<P>(v);
		}
		r = padd<P>(r, integrate_edge2<P>(prev, cur));
		prev = cur;
		cur = next;
	}
	r = padd<P>(r, integrate_edge2<P>(prev, first));
	const uint32_t all = (1u << n) - 1u;
	float integral[2];
	bool away[2];
	const uint32_t above[2] = {above_s, above_c};
	const float sum[2] = {r.x, r.y};
#pragma unroll
	for (int s = 0; s != 2; ++s) {
		float rs = sum[s];
		bool a = false;
		if (above[s] == all) {
			rs = fabsf(rs);
		} else if (above[s] == 0) {
			rs = 0.0f;
			a = true;
		} else {
			bool unused = true;
			rs = clipped_integral<P, false>(load_matrix(f, s), record, n, above[s], unused);
			a = rs < 0.0f;
			rs = a ? 0.0f : rs;
		}
		integral[s] = rs;
		away[s] = a;
	}
	const f3 radiance = mk3(head.x, head.y, head.z);
	f3 result = splat(0.0f);
	const f3 diffuse = away[0] ? splat(0.0f) : mul(scale(mk3(f0.x, f0.y, f0.z), integral[0]), radiance);
	result = add(result, diffuse);
	const f3 ggx = away[1] ? splat(0.0f) : mul(splat(integral[1] * f0.w), radiance);
	const f3 color = add(result, ggx);
	p_hat = P::sqrt(dot(color, color));
}

// The first pass's operations per numerics mode.  Both return sums and
// quotients of one sign throughout (see candidate_first_pass).
//
// Exact numerics keeps every normalised vertex negated: the reciprocal of -s
// gives Markstein's correction without a sign change, and dot and cross
// products of two negated vertices equal those of the vertices.  The edge
// integral's quotient is negated in the same way, so the sum is the negated
// sum, whose magnitude is what is kept.
struct FirstPassExact {
	PairExact o;
	RL_DEV explicit FirstPassExact(float neg_zero) : o{pair(neg_zero)} {}
	RL_DEV float2 row(float2 c0, float2 c1, float2 c2, float2 c3, float2 px, float2 py, float2 pz) const {
		return o.add(o.add(o.add(o.mul(c0, px), o.mul(c1, py)), o.mul(c2, pz)), c3);
	}
	RL_DEV float2 dot(const f3x2& a, const f3x2& b) const {
		return o.add(o.add(o.mul(a.x, b.x), o.mul(a.y, b.y)), o.mul(a.z, b.z));
	}
	RL_DEV f3x2 normalized(const f3x2& v, float2 d) const {
		const float2 nr = rsqrt_negated(o, d);
		return {o.mul(v.x, nr), o.mul(v.y, nr), o.mul(v.z, nr)};
	}
	// r + the edge integral of a, b, whose dot product is x.
	RL_DEV float2 add_edge(float2 r, const f3x2& a, const f3x2& b, float2 x) const {
		return o.add(r, o.mul(o.sub(o.mul(a.x, b.y), o.mul(a.y, b.x)), edge_fit_negated(o, x)));
	}
};
// Fast numerics: fused multiply-adds, the hardware's reciprocal square root
// and quotient.
struct FirstPassFast {
	RL_DEV explicit FirstPassFast(float) {}
	RL_DEV float2 row(float2 c0, float2 c1, float2 c2, float2 c3, float2 px, float2 py, float2 pz) const {
		return __fadd2_rn(__ffma2_rn(c2, pz, __ffma2_rn(c1, py, __fmul2_rn(c0, px))), c3);
	}
	RL_DEV float2 dot(const f3x2& a, const f3x2& b) const {
		return __ffma2_rn(a.z, b.z, __ffma2_rn(a.y, b.y, __fmul2_rn(a.x, b.x)));
	}
	RL_DEV f3x2 normalized(const f3x2& v, float2 d) const {
		const float2 s = make_float2(rsqrt_approx(d.x), rsqrt_approx(d.y));
		return {__fmul2_rn(v.x, s), __fmul2_rn(v.y, s), __fmul2_rn(v.z, s)};
	}
	RL_DEV float2 add_edge(float2 r, const f3x2& a, const f3x2& b, float2 x) const {
		const float2 num = __ffma2_rn(__ffma2_rn(pair(0.0145206f), x, pair(0.4965155f)), x, pair(0.8543985f));
		const float2 den = __ffma2_rn(__fadd2_rn(pair(4.1616724f), x), x, pair(3.4175940f));
		const float2 t = __fmul2_rn(num, make_float2(rcp_approx(den.x), rcp_approx(den.y)));
		const float2 ay = make_float2(-a.y.x, -a.y.y);
		return __ffma2_rn(__ffma2_rn(a.x, b.y, __fmul2_rn(ay, b.x)), t, r);
	}
};
template <class P> struct FirstPass {
	using type = FirstPassExact;
};
template <> struct FirstPass<FastNumerics> {
	using type = FirstPassFast;
};

// The first pass: one candidate with no branch in its vertex loop but the
// loop's.  False (the caller defers the item, which is then clipped) when a
// space clips the polygon partially, a squared length lies outside the square
// root's range or an edge spans 90 degrees or more.
template <class O>
RL_DEV bool candidate_first_pass(const float4* f, const float4* record, float neg_zero, float& p_hat) {
	const O o(neg_zero);
	const RecordWords head = load_words(record);  // {radiance, vertex count}, vertex 0
	RecordWords q = load_words(record + kRecordVertex + 1);  // vertices 1 and 2
	const uint32_t n = __float_as_uint(head.a.w);
	float2 r = pair(0.0f);
	// What decides whether the branch-free forms apply: the least squared
	// length (an infinite or NaN one leaves a NaN sum), the least cosine of an
	// edge, the least z of both spaces and the greatest of each (as signed
	// words, ordered like the floats where both are positive; -0 counts as
	// below, +0 as not above).
	uint32_t d_min = 0xffffffffu;
	int32_t x_min = 0x7fffffff, z_min = 0x7fffffff, zs_max = INT32_MIN, zc_max = INT32_MIN;
	auto edge = [&](const f3x2& a, const f3x2& b) {
		const float2 x = o.dot(a, b);
		x_min = __vimin3_s32(x_min, __float_as_int(x.x), __float_as_int(x.y));
		r = o.add_edge(r, a, b, x);
	};
	const mat43x2 t = load_pairs(f);
	auto vertex = [&](float4 p) -> f3x2 {  // transformed and normalised
		const float2 px = pair(p.x), py = pair(p.y), pz = pair(p.z);
		const f3x2 v = {o.row(t.c[0].x, t.c[1].x, t.c[2].x, t.c[3].x, px, py, pz),
		                o.row(t.c[0].y, t.c[1].y, t.c[2].y, t.c[3].y, px, py, pz),
		                o.row(t.c[0].z, t.c[1].z, t.c[2].z, t.c[3].z, px, py, pz)};
		z_min = __vimin3_s32(z_min, __float_as_int(v.z.x), __float_as_int(v.z.y));
		zs_max = max(zs_max, __float_as_int(v.z.x));
		zc_max = max(zc_max, __float_as_int(v.z.y));
		const float2 d = o.dot(v, v);
		d_min = __vimin3_u32(d_min, __float_as_uint(d.x), __float_as_uint(d.y));
		return o.normalized(v, d);
	};
	const f3x2 first = vertex(head.b);
	f3x2 a = vertex(q.a), b;
	edge(first, a);
#pragma unroll 1
	for (uint32_t j = 2;; j += 2) {
		// Vertex j is in q.b; the next two are fetched while it is used.
		RecordWords next = q;
		if (j + 1 < n) next = load_words(record + kRecordVertex + 1 + j);
		b = vertex(q.b);
		edge(a, b);
		if (j + 1 >= n) break;
		a = vertex(next.a);
		edge(b, a);
		if (j + 2 >= n) {
			b = a;
			break;
		}
		q.b = next.b;
	}
	edge(b, first);
	const bool below_s = zs_max <= 0, below_c = zc_max <= 0;
	if (!(d_min >= kRootMin && x_min > 0 && (z_min > 0 || (below_s && below_c)))) return false;
	const f3 radiance = mk3(head.a.x, head.a.y, head.a.z);
	const float4 f0 = f[0];
	const f3 diffuse = below_s ? splat(0.0f) : mul(scale(mk3(f0.x, f0.y, f0.z), fabsf(r.x)), radiance);
	const f3 ggx = below_c ? splat(0.0f) : mul(splat(fabsf(r.y) * f0.w), radiance);
	const f3 color = add(add(splat(0.0f), diffuse), ggx);
	bool ok = true;
	p_hat = sqrt_checked<ExactNumerics>(dot(color, color), ok);
	return ok;
}

// A deferred candidate, clipped where it has to be.  Exact numerics: the
// scalar forms, branch-free where they apply, the general ones otherwise.
// Fast numerics: the paired form.
template <class P> RL_DEV void deferred_candidate(const float4* f, const float4* record, float& p_hat) {
	if (!binned_candidate<P, true>(f, record, p_hat)) binned_candidate<P, false>(f, record, p_hat);
}
template <> RL_DEV void deferred_candidate<FastNumerics>(const float4* f, const float4* record, float& p_hat) {
	binned_candidate_pair<FastNumerics>(f, record, p_hat);
}

// The reservoir's test rnd < w / w_sum (insert_in_reservoir) for w > 0: the
// division is needed only where t = rnd * w_sum lies within 2^-20 of w, or out
// of the range in which t and w / w_sum are sure to be normal numbers.  With t
// normal, t < w means a quotient above rnd, which is a multiple of 2^-32 and not
// 0 then; t > w means that the rounded quotient, however small, is below rnd.
// (A rnd of 0 is refused only where the quotient underflows to 0: it divides.)
template <class P> RL_DEV bool reservoir_accepts(float rnd, float w, float w_sum) {
	const float t = rnd * w_sum;
	const bool normal = t > 1e-25f && w_sum < 1e30f;
	if (normal && t < w * (1.0f - 0x1p-20f)) return true;
	if (normal && t > w * (1.0f + 0x1p-20f)) return false;
	return rnd < P::div(w, w_sum);
}

// One warp tile t (pixels t * kPixels .. + kPixels - 1) of one frame set:
// candidates, evaluation, replay and reservoir records for all frames.
// tile is the warp's shared-memory tile, phat its p_hat slot.
template <class P, int kPixels, int kChunk>
RL_DEV void binned_tile(const RisParams& pr, WarpTile<BinnedSuper<P>::value, kPixels, kChunk>& tile, float* phat,
                        uint32_t t) {
	constexpr int kSuper = BinnedSuper<P>::value;
	const uint32_t lane = threadIdx.x % 32;
	const uint32_t np = pr.width * pr.height;
	const int n_lights = pr.scene.light_count;
	// Lanes kPixels..31 own no pixel: they draw nothing and only evaluate
	// items of the sorted lists.
	const bool own = lane < (uint32_t) kPixels;
	const uint32_t i = t * kPixels + lane;
	const bool valid = own && i < np && !(pr.primitive && pr.primitive[i] == 0xffffffffu);
	if (valid) {
		const float* g = pr.gbuffer;
		const size_t snp = np;
		const f3 position = mk3(g[0 * snp + i], g[1 * snp + i], g[2 * snp + i]);
		const f3 normal = mk3(g[3 * snp + i], g[4 * snp + i], g[5 * snp + i]);
		const f3 outgoing = mk3(g[6 * snp + i], g[7 * snp + i], g[8 * snp + i]);
		const f3 fresnel_0 = mk3(g[13 * snp + i], g[14 * snp + i], g[15 * snp + i]);
		const float roughness = g[16 * snp + i];
		const f3 diffuse_albedo = mk3(g[10 * snp + i], g[11 * snp + i], g[12 * snp + i]);
		const float fl = dot(fresnel_0, mk3(0.2126f, 0.7152f, 0.0722f));
		const Ltc ltc = get_ltc_coefficients<P>(pr.scene, fl, roughness, position, normal, outgoing);
		store_frame(tile.frame[lane], diffuse_albedo, ltc.albedo, ltc.world_to_shading,
		            mul(ltc.shading_to_cosine, ltc.world_to_shading));
	}
	// Background is noted by one of its lanes, and nothing waits for that.
	if (pr.compact && own && i < np && !valid && lane == (uint32_t) __ffs(__activemask()) - 1u)
		atomicOr(&pr.counters->background, 1u);
	if (lane == 0) tile.deferred_count = 0;
	__syncwarp();
	// The noise state at the start of frame f (get_noise_accessor with the
	// frame's random offset).
	auto frame_seed = [&](uint32_t f) -> uint32_t {
		if (!valid) return 0u;
		const uint32_t rn_x = pr.animate ? wang_random_number((pr.noise_seed + f) * 4u) : 0u;
		return get_noise_accessor(i % pr.width, i / pr.width, pr.width, rn_x);
	};
	auto drawn_light = [&](float u) -> int {
		const int idx = (int) (u * (float) n_lights);
		return idx > n_lights - 1 ? n_lights - 1 : idx;
	};
	// The tile's work comes in units of one frame's super-chunk.  Up to
	// kWindow units are evaluated before their reservoirs are replayed, so
	// that deferred items of several units share the general path's rounds:
	// unit u of the window keeps its p_hat values at phat[u * kUnitSlots +
	// slot].
	constexpr uint32_t kUnitSlots = (uint32_t) (kPixels * kSuper);
	constexpr uint32_t kWindow = (uint32_t) kPHatSlot / kUnitSlots;
	const uint32_t units_per_frame = ((uint32_t) pr.candidate_count + kSuper - 1) / kSuper;
	const uint32_t units = pr.frame_count * units_per_frame;
	uint32_t window = 0;  // units evaluated since the last replay
	uint32_t draw = 0;    // the draw phase's noise state
	for (uint32_t unit = 0; unit != units; ++unit) {
		const uint32_t f = unit / units_per_frame, cs = (unit % units_per_frame) * kSuper;
		if (cs == 0) draw = frame_seed(f);
		const int super_count = min(kSuper, pr.candidate_count - (int) cs);
		const bool window_ends = window + 1 == kWindow || unit + 1 == units;
		float* const uphat = phat + window * kUnitSlots;
		for (int c0 = 0; c0 < super_count; c0 += kChunk) {
			const int chunk = min(kChunk, super_count - c0);
			// 1. This lane's candidate lights, counted by vertex count in six
			//    10-bit fields of a word (field b: b + 3 vertices).
			int light[kChunk];
			uint32_t field[kChunk];  // the field's shift
			unsigned long long counts = 0;
#pragma unroll
			for (int k = 0; k != kChunk; ++k) {
				light[k] = -1;
				field[k] = 0;
				if (valid && k < chunk) {
					int idx = drawn_light(get_noise_1(draw));
					if (pr.candidates)
						idx = pr.candidates[((size_t) f * np + i) * pr.candidate_count + cs + c0 + k].light;
					draw = 1664525u * draw + 1013904223u;  // the reservoir's draw
					light[k] = idx;
					field[k] = 10u * (light_vertex_count(pr.scene, idx) - 3u);
					counts += 1ull << field[k];
				}
			}
			// 2. Counting sort: a scan of the fields across the warp gives
			//    each lane's place in every bin, and one multiplication adds
			//    the bins' starts (field b of totals * (2^10 + ... + 2^50) is
			//    the sum of the fields below b; no field reaches 1024).
			unsigned long long place = counts;
#pragma unroll
			for (int d = 1; d < 32; d <<= 1) {
				const unsigned long long o = __shfl_up_sync(0xffffffffu, place, d);
				if ((int) lane >= d) place += o;
			}
			const unsigned long long totals = __shfl_sync(0xffffffffu, place, 31);
			const unsigned long long starts = totals * 0x0004010040100400ull;
			const uint32_t item_count = (uint32_t) ((starts >> 50) & 1023u) + (uint32_t) ((totals >> 50) & 1023u);
			place += starts - counts;
#pragma unroll
			for (int k = 0; k != kChunk; ++k) {
				if (light[k] >= 0) {
					tile.item[(uint32_t) (place >> field[k]) & 1023u] =
					    ((uint32_t) light[k] << 10) | ((c0 + k) * kPixels + lane);
					place += 1ull << field[k];
				}
			}
			__syncwarp();
			// 3. Evaluate the sorted items, 32 at a time; defer partial clips
			//    (with their unit).
			for (uint32_t base = 0; base < item_count; base += 32) {
				const uint32_t it = base + lane;
				if (it < item_count) {
					const uint32_t item = tile.item[it];
					const uint32_t slot = item & 1023u;
					float ph;
					if (candidate_first_pass<typename FirstPass<P>::type>(
					        tile.frame[slot % kPixels], light_record(pr.scene, (int) (item >> 10)), pr.neg_zero, ph)) {
						uphat[slot] = ph;
					} else {
						const uint32_t d = atomicAdd(&tile.deferred_count, 1u);
						tile.deferred[d] = item;
						tile.deferred_unit[d] = (uint8_t) window;
					}
				}
			}
			__syncwarp();
			// Deferred items 32 at a time; the rest when the window ends.
			const uint32_t least = window_ends && c0 + kChunk >= super_count ? 1u : 32u;
			for (uint32_t pending = tile.deferred_count; pending >= least;) {
				const uint32_t take = min(pending, 32u);
				pending -= take;
				if (lane < take) {
					const uint32_t d = pending + lane;
					const uint32_t item = tile.deferred[d], slot = item & 1023u;
					float ph = 0.0f;
					deferred_candidate<P>(tile.frame[slot % kPixels], light_record(pr.scene, (int) (item >> 10)), ph);
					phat[tile.deferred_unit[d] * kUnitSlots + slot] = ph;
				}
				__syncwarp();
				if (lane == 0) tile.deferred_count = pending;
				__syncwarp();
			}
		}
		++window;
		if (!window_ends) continue;
		// 4. Reservoir updates of the window's units in candidate order,
		//    drawing the same noise again.  A frame whose super-chunks reach
		//    past the window leaves its reservoir in its record.
		const float p = P::rcp((float) n_lights);
		// With uniform candidates and a power-of-two light count, p is a power
		// of two and p_hat / p equals p_hat * (1 / p) bit for bit (scaling by a
		// power of two is exact): the replay multiplies instead of dividing.
		const bool scale_weight = !pr.candidates && (n_lights & (n_lights - 1)) == 0;
		const float inv_p = (float) n_lights;
		uint32_t seed = 0;
		float w_sum = 0.0f, sample_value = 0.0f;
		int res_index = -1;
		for (uint32_t u = 0; u != window; ++u) {
			const uint32_t ru = unit + 1 - window + u;
			const uint32_t rf = ru / units_per_frame, rcs = (ru % units_per_frame) * kSuper;
			const size_t at = (size_t) rf * np + i;
			if (rcs == 0) {
				seed = frame_seed(rf);
				w_sum = 0.0f;
				sample_value = 0.0f;
				res_index = -1;
			} else if (u == 0 && valid) {
				const ReservoirRecord r = pr.records[at];
				res_index = r.light_index;
				w_sum = r.w_sum;
				sample_value = r.p_hat;
				seed = r.seed;
			}
			const int rcount = min(kSuper, pr.candidate_count - (int) rcs);
			const float* const rphat = phat + u * kUnitSlots + lane;
			if (valid) {
				int chosen = -1;           // the candidate that the reservoir took last,
				uint32_t chosen_seed = 0;  // and the noise state that drew its light
#pragma unroll 4
				for (int k = 0; k < rcount; ++k) {
					seed = 1664525u * seed + 1013904223u;  // the light's draw
					const uint32_t light_seed = seed;
					const float rnd = get_noise_1(seed);
					const float p_hat = rphat[k * kPixels];
					float pk = p;
					if (pr.candidates) pk = pr.candidates[at * pr.candidate_count + rcs + k].pdf;
					const float w = scale_weight ? p_hat * inv_p : P::div(p_hat, pk);
					if (pr.train_stride && rf == 0 && i % pr.train_stride == pr.train_phase)
						pr.train_candidates[(size_t) i * pr.candidate_count + rcs + k].pdf = w;
					w_sum += w;
					if (w > 0.0f && reservoir_accepts<P>(rnd, w, w_sum)) {
						chosen = k;
						chosen_seed = light_seed;
						sample_value = p_hat;
					}
				}
				if (chosen >= 0)
					res_index = pr.candidates ? pr.candidates[at * pr.candidate_count + rcs + chosen].light
					                          : drawn_light(__uint2float_rn(chosen_seed) * 2.3283064365386962890625e-10f);
			}
			if (u + 1 == window || rcs + kSuper >= (uint32_t) pr.candidate_count) {
				if (valid)
					pr.records[at] = ReservoirRecord{res_index, w_sum, sample_value, seed};
				else if (own && i < np)
					pr.records[at] = ReservoirRecord{-1, 0.0f, 0.0f, 0u};
			}
		}
		window = 0;
		__syncwarp();
	}
	__syncwarp();
}

template <class P, int kPixels, int kChunk>
__global__ void __launch_bounds__(32 * kBinnedWarps, BinnedMinBlocks<P>::value)
ris_candidates_binned_kernel(const __grid_constant__ RisParams pr) {
	extern __shared__ __align__(16) unsigned char smem_raw[];
	allow_next();
	using Tile = WarpTile<BinnedSuper<P>::value, kPixels, kChunk>;
	Tile& tile = reinterpret_cast<Tile*>(smem_raw)[threadIdx.x / 32];
	float* const phat = pr.p_hat_scratch + (size_t) (blockIdx.x * kBinnedWarps + threadIdx.x / 32) * kPHatSlot;
	const uint32_t tiles = (pr.width * pr.height + kPixels - 1) / kPixels;
	// (In fast numerics the cursor alone is 0.6% faster on large frames.)
	if constexpr (std::is_same<P, FastNumerics>::value) {
		for (uint32_t t = next_warp_tile(&pr.counters->tile); t < tiles; t = next_warp_tile(&pr.counters->tile))
			binned_tile<P, kPixels, kChunk>(pr, tile, phat, t);
	} else {
		for_warp_tiles(&pr.counters->tile, tiles, [&](uint32_t t) { binned_tile<P, kPixels, kChunk>(pr, tile, phat, t); });
	}
}

template <class P, int kPixels, int kChunk> constexpr size_t binned_smem_bytes() {
	return sizeof(WarpTile<BinnedSuper<P>::value, kPixels, kChunk>) * kBinnedWarps;
}

// First launch of a candidate kernel on a device: raises its shared-memory
// limit (above the 48 KB available without opting in) and stores in
// resident[device] the blocks that fit on the device at once (resident
// blocks per SM times the SM count), the kernel's persistent grid: one wave
// whose warps take tiles from the launch's cursor until none is left.  Done once
// per device, so that later launches, including those captured into a CUDA
// graph, make no other runtime call.
template <class Kernel>
cudaError_t configure_candidate_kernel(Kernel kernel, size_t smem, std::atomic<uint64_t>& configured,
                                       std::atomic<int>* resident, int& device) {
	cudaError_t e = cudaGetDevice(&device);
	if (e != cudaSuccess) return e;
	const uint64_t bit = 1ull << (device & 63);
	if (configured.load() & bit) return cudaSuccess;
	e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
	int sms = 0, per_sm = 0;
	if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
	if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * kBinnedWarps, smem);
	if (e != cudaSuccess) return e;
	resident[device & 63].store(std::max(1, sms * std::min(per_sm, kCandidateBlocksPerSm)));
	configured.fetch_or(bit);
	return cudaSuccess;
}

// Launches the binned candidate kernel.  Its shared memory exceeds the 48 KB
// available without opting in, so the limit is raised the first time the
// kernel runs on a device (once, so that later launches, including those
// captured into a CUDA graph, make no other runtime call).
// grid_cap is the largest grid the p_hat scratch has warp slots for.
template <class P, int kPixels, int kChunk>
cudaError_t launch_candidates_binned(const RisParams& p, cudaStream_t stream, int grid_cap) {
	const size_t pixels = (size_t) p.width * p.height;
	const size_t blocks = (pixels + kPixels * kBinnedWarps - 1) / (kPixels * kBinnedWarps);
	const int grid = (int) std::max<size_t>(1, std::min<size_t>(blocks, (size_t) grid_cap));
	// Without p_hat scratch (the allocation-free entry point), the kernel with
	// one thread per pixel computes the same records.
	if (!p.p_hat_scratch) {
		ris_candidates_kernel<P><<<grid_for_pixels(pixels, grid_cap), 128, 0, stream>>>(p);
		return cudaGetLastError();
	}
	static std::atomic<uint64_t> configured{0};
	static std::atomic<int> resident[64];
	int device = 0;
	const cudaError_t e = configure_candidate_kernel(ris_candidates_binned_kernel<P, kPixels, kChunk>,
	                                                 binned_smem_bytes<P, kPixels, kChunk>(), configured, resident, device);
	if (e != cudaSuccess) return e;
	ris_candidates_binned_kernel<P, kPixels, kChunk>
	    <<<std::min(grid, resident[device & 63].load()), 32 * kBinnedWarps, binned_smem_bytes<P, kPixels, kChunk>(),
	       stream>>>(p);
	return cudaGetLastError();
}

}  // namespace risltc
