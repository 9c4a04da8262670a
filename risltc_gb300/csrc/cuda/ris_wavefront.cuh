// ris_wavefront.cuh - the shading phase of the two-kernel pipeline with its
// shadow rays traced in a separate pass:
//
//   ris_sample_kernel: per pixel and frame, the estimator of
//     evaluate_polygonal_light_shading_peters (shading_pass.frag.glsl:292-397)
//     for the chosen light up to the visibility test.  For each of its (at
//     most two) samples it stores the MIS-weighted contribution for both
//     outcomes of the shadow ray and puts the ray at the sample's own place
//     in the queue.  Nearly every sample of a surface has one; where there is
//     none the place holds an empty interval.  In large calls background has
//     no places (queue_covered).  In this order a warp traces both rays
//     of 16 neighbouring pixels: grouped by light (a counting sort, 0.68 ms
//     of its own) they took 4.39 ms per 4-frame 1080p launch with 16,384
//     lights, appended technique by technique 4.36, in this order 4.10 (3.36
//     with the traversal's present form).
//   shadow_trace_kernel, and shadow_trace_shares_kernel for large calls: one
//     any-hit query per queued ray, with a small register footprint and no
//     divergence from the shading code around it.
//   ris_resolve_kernel: per pixel, picks each sample's contribution by its
//     ray's outcome and finishes the frame and the accumulation exactly as
//     ris_shade_kernel does.
// The contributions are the same operations on the same values, added in
// the same order, so the pixels are bit-identical to ris_shade_kernel's.
// ris_estimate_kernel: the sample and resolve phases in one where no shadow ray is
// traced.
// Used for one sample per technique (SAMPLE_COUNT == 1, the reference's
// default) with shadows on: after the candidate kernel, or (uniform_light)
// with one uniformly drawn light per pixel-frame, the reference's ground-truth
// estimator, for which shade_kernel with its inline rays took 17.6 ms per
// 4-frame 640x360 call with 5,000 occluders against 1.05 here.
// Restates upstream risltc routines (GPLv3): see NOTICE.
#pragma once
#include "ris_kernels.cuh"

namespace risltc {

// Per-sample mode, two bits per technique j in SampleRecord::flags.
enum : uint32_t {
	kSampleSkip = 0,    // no contribution (dir.z <= 0 or no such sample)
	kSampleFixed = 1,   // contribution c[j][0], no ray needed
	kSampleTraced = 2,  // c[j][0] if the ray is unoccluded, else c[j][1]
	kSampleNoLight = 1u << 8,  // empty reservoir: the frame's colour is zero
};

// The estimator's state between the sample and resolve kernels (64 bytes).
struct SampleRecord {
	float c[2][2][3];  // [technique][unoccluded, occluded][rgb]
	float W;           // the reservoir's unbiased contribution weight
	uint32_t flags;
	uint32_t number;   // the pixel's in the queue
	uint32_t pad;
};
static_assert(sizeof(SampleRecord) == 64, "SampleRecord layout");

// A shadow ray: origin, direction and t_max (t_min is get_polygon_visibility's
// 1e-3).
struct ShadowRay {
	float4 origin;
	float4 dir_tmax;
};
// No ray at a covered pixel's place: t_max below t_min, so that the query ends at
// the root's box.
RL_DEV void store_no_ray(ShadowRay* ray) {
	ray->origin = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
	ray->dir_tmax = make_float4(0.0f, 0.0f, 1.0f, -1.0f);
}

// The queue's places are [frame][number][technique], with room for `pixels`
// numbers in a frame.  A pixel's number is its index, and with background in the
// G-buffer (noted by the candidate kernel) the covered pixels, those that are no
// background, are numbered as the sample kernel's warps come to them, so that
// background costs nothing.  (Numbered in every call, full frames took 0.3 to
// 0.8% longer.)  Whether they are, and the pixels that have places:
RL_DEV bool has_numbers(const RisParams& pr) { return pr.compact && pr.counters->background != 0; }
RL_DEV uint32_t queue_covered(const LaunchCounters* counters, uint32_t pixels) {
	return counters->background != 0 ? counters->covered : pixels;
}
// The place of ray g of the call:
RL_DEV uint32_t queue_place(uint32_t g, uint32_t covered, uint32_t pixels) {
	return covered == pixels ? g : g + g / (2u * covered) * (2u * (pixels - covered));
}

// Technique j's two contributions (unoccluded, occluded) into floats
// 6j .. 6j + 5 of a sample record.
RL_DEV void store_contributions(SampleRecord* dst, int j, f3 c0, f3 c1) {
	float* f = reinterpret_cast<float*>(dst);
	if (j == 0) {
		*reinterpret_cast<float4*>(f) = make_float4(c0.x, c0.y, c0.z, c1.x);
		*reinterpret_cast<float2*>(f + 4) = make_float2(c1.y, c1.z);
	} else {
		*reinterpret_cast<float2*>(f + 6) = make_float2(c0.x, c0.y);
		*reinterpret_cast<float4*>(f + 8) = make_float4(c0.z, c1.x, c1.y, c1.z);
	}
}

// evaluate_polygonal_light_shading_peters or, with peters false, the PSA
// branch of evaluate_polygonal_light_shading, for SAMPLE_COUNT == 1 up to the
// visibility test.  Gives sink(j, unoccluded, occluded) technique j's
// contributions (zero where it has none) and, with kRays, writes each traced
// technique's shadow ray into rays[j], as soon as they are known, and returns
// the techniques' modes (without kRays none is traced).  l is the light whose
// device record is `record`; poly is the thread's polygon buffer.
template <class P, bool kRays, class Sink>
RL_DEV uint32_t psa_mis_emit(const ShadeParams& pr, bool peters, const ShadingData& sd, Ltc ltc, const Light& l,
                             const float4* record, uint32_t& seed, Sink sink, ShadowRay* rays, PsaPolygon& poly) {
	const bool fa = pr.fast_atan != 0;
	const bool biased = pr.technique == sample_polygon_projected_solid_angle_biased;
	side_flip(ltc, sd, l);
	// One polygon buffer serves both spaces: the shading-space polygon is
	// prepared and sampled, then the cosine-space one is prepared into the
	// same storage and sampled (if it has a projected solid angle).  The
	// samples draw the noise in the reference's order (diffuse, then
	// specular), and after sampling only the projected solid angles are
	// needed, so the values equal those of psa_prepare_both followed by both
	// samples.
	float psa[2] = {0.0f, 0.0f};
	int technique_count = 1;
	f3 dir_d = mk3(0.0f, 0.0f, 1.0f), dir_s = mk3(0.0f, 0.0f, 1.0f);
#pragma unroll 1
	for (int j = 0; j != 2; ++j) {
		const uint32_t vc = prepare_space_record<P>(j == 0 ? ltc.world_to_shading
		                                                  : mul(ltc.shading_to_cosine, ltc.world_to_shading),
		                                           record, l.vertex_count, poly, fa);
		psa[j] = vc == 0 ? 0.0f : poly.psa;
		if (j == 0 && (vc == 0 || psa[0] == 0.0f)) {
			sink(0, splat(0.0f), splat(0.0f));
			sink(1, splat(0.0f), splat(0.0f));
			return 0;
		}
		if (j == 1 && !(psa[1] > 0.0f)) break;
		const f3 dir = sample_psa<P>(poly, get_noise_2(seed), fa, biased);
		if (j == 0) {
			dir_d = dir;
		} else {
			dir_s = normalize<P>(mul(ltc.cosine_to_shading, dir));
			technique_count = 2;
		}
	}
	float specular_weight = ltc.albedo * psa[1];
	f3 diffuse_weight = scale(max3(sd.diffuse_albedo, splat(0.01f)), psa[0]);
	float rcp_d = P::rcp(psa[0]);
	float rcp_s = P::rcp(psa[1]);
	f3 specular_weight_rgb = splat(specular_weight);
	if (pr.mis_heuristic == mis_heuristic_optimal) {
		f3 rop = scale(l.radiance, kInvPi);
		diffuse_weight = mul(diffuse_weight, rop);
		specular_weight_rgb = mul(specular_weight_rgb, rop);
	}
	const bool shadows = kRays && pr.shadows && pr.scene.triangle_count != 0;
	uint32_t modes = 0;
#pragma unroll 1
	for (int j = 0; j != 2; ++j) {
		f3 dir = (j == 0) ? dir_d : dir_s;
		if (j >= technique_count || dir.z <= 0.0f) {
			sink(j, splat(0.0f), splat(0.0f));
			continue;
		}
		float diffuse_density = dir.z * rcp_d;
		float specular_density = evaluate_ltc_density<P>(ltc, dir, rcp_s);
		f3 world_dir = transpose_mul(ltc.world_to_shading, dir);
		const bool side = dot(sd.normal, world_dir) > 0.0f;
		const bool traced = side && shadows;
		const f3 rb_lit = side ? mul(l.radiance, evaluate_brdf<P>(sd, world_dir)) : splat(0.0f);
		// This technique's weight and density first, the other's second.
		const f3 own_weight = j == 0 ? diffuse_weight : specular_weight_rgb;
		const f3 other_weight = j == 0 ? specular_weight_rgb : diffuse_weight;
		const float own_density = j == 0 ? diffuse_density : specular_density;
		const float other_density = j == 0 ? specular_density : diffuse_density;
		// Outcome 0: visible iff side (unoccluded or untraced); outcome 1:
		// occluded.
		f3 c[2] = {splat(0.0f), splat(0.0f)};
#pragma unroll 1
		for (int o = 0; o != (traced ? 2 : 1); ++o) {
			const bool visibility = (o == 0) ? side : false;
			f3 integrand = scale(visibility ? rb_lit : splat(0.0f), dir.z);
			f3 r;
			if (j == 0 && psa[1] <= 0.0f)
				r = visibility || !peters ? scale(integrand, P::rcp(diffuse_density)) : splat(0.0f);
			else
				r = mis_estimate<P>(pr.mis_heuristic, integrand, own_weight, own_density, other_weight, other_density,
				                    pr.mis_visibility_estimate);
			if (o == 0) c[0] = r; else c[1] = r;
		}
		sink(j, c[0], c[1]);
		if (kRays && traced) {
			// get_polygon_visibility, shading_pass.frag.glsl:112-129
			float max_t = P::div(-plane_dot(sd.position, l.plane),
			                     world_dir.x * l.plane[0] + world_dir.y * l.plane[1] + world_dir.z * l.plane[2]);
			max_t -= 1e-3f;
			rays[j] = ShadowRay{make_float4(sd.position.x, sd.position.y, sd.position.z, 0.0f),
			                    make_float4(world_dir.x, world_dir.y, world_dir.z, max_t)};
		}
		modes |= (traced ? kSampleTraced : kSampleFixed) << (2 * j);
	}
	return modes;
}

RL_DEV void store_sample(SampleRecord* dst, const f3 (&c)[2][2], float W, uint32_t flags) {
	float4* q = reinterpret_cast<float4*>(dst);
	q[0] = make_float4(c[0][0].x, c[0][0].y, c[0][0].z, c[0][1].x);
	q[1] = make_float4(c[0][1].y, c[0][1].z, c[1][0].x, c[1][0].y);
	q[2] = make_float4(c[1][0].z, c[1][1].x, c[1][1].y, c[1][1].z);
	q[3] = make_float4(W, __uint_as_float(flags), 0.0f, 0.0f);
}

// Pixel i's shading data and LTC frame.
template <class P> RL_DEV void load_pixel(const RisParams& pr, uint32_t i, ShadingData& sd, Ltc& ltc) {
	const float* g = pr.gbuffer;
	const size_t snp = pr.width * pr.height;
	sd.position = mk3(g[0 * snp + i], g[1 * snp + i], g[2 * snp + i]);
	sd.normal = mk3(g[3 * snp + i], g[4 * snp + i], g[5 * snp + i]);
	sd.outgoing = mk3(g[6 * snp + i], g[7 * snp + i], g[8 * snp + i]);
	sd.lambert_outgoing = g[9 * snp + i];
	sd.diffuse_albedo = mk3(g[10 * snp + i], g[11 * snp + i], g[12 * snp + i]);
	sd.fresnel_0 = mk3(g[13 * snp + i], g[14 * snp + i], g[15 * snp + i]);
	sd.roughness = g[16 * snp + i];
	const float fl = dot(sd.fresnel_0, mk3(0.2126f, 0.7152f, 0.0722f));
	ltc = get_ltc_coefficients<P>(pr.scene, fl, sd.roughness, sd.position, sd.normal, sd.outgoing);
}

#ifndef RISLTC_SAMPLE_MIN_BLOCKS
#define RISLTC_SAMPLE_MIN_BLOCKS 4
#endif
// Threads per block of the sample kernels.  Each thread's PSA polygon buffer
// (196 bytes, indexed by the sorting network and the sector search) is a
// slot of a shared-memory array: slots are 49 words apart, so the lanes'
// words of one index fall in 32 distinct banks.  In local memory the 16
// resident warps' buffers (about 240 KB per SM) did not stay in L1 (sample
// kernel 5.71 ms per 4-frame 1080p launch, 4.14 ms with the shared slots).
constexpr int kSampleThreads = 128;
// The sample phase of pixel i (all frames of the call), called by whole warps;
// i may be past the frame (the thread then does nothing).
// kUniform: RisParams::uniform_light (a variant of its own: its few
// instructions cost the other 2%).
template <class P, bool kUniform>
RL_DEV void sample_pixel(const RisParams& pr, uint32_t i, PsaPolygon& poly, bool numbered) {
	const uint32_t np = pr.width * pr.height;
	ShadeParams sp;  // the fields psa_prepare_both and psa_mis_emit read
	sp.scene = pr.scene;
	sp.technique = kUniform ? pr.technique : (int) sample_polygon_ltc_cp;
	const bool peters = !kUniform || pr.technique == sample_polygon_ltc_cp;
	sp.mis_heuristic = pr.mis_heuristic;
	sp.sample_count = 1;
	sp.mis_visibility_estimate = pr.mis_visibility_estimate;
	sp.fast_atan = pr.fast_atan;
	sp.shadows = pr.shadows;
	sp.error = pr.error;
	{
		const bool active = i < np && !(pr.primitive && pr.primitive[i] == 0xffffffffu);
		uint32_t number = i;
		if (numbered) {
			const uint32_t covered = __ballot_sync(0xffffffffu, active);
			if (threadIdx.x % 32 == 0 && covered) number = atomicAdd(&pr.counters->covered, (uint32_t) __popc(covered));
		}
		ShadingData sd;
		Ltc ltc;
		if (active) {
			load_pixel<P>(pr, i, sd, ltc);
		}
		if (numbered)
			number = __shfl_sync(0xffffffffu, number, 0) +
			         (uint32_t) __popc(__ballot_sync(0xffffffffu, active) & ((1u << threadIdx.x % 32) - 1u));
		for (uint32_t f = 0; f != pr.frame_count; ++f) {
			const size_t pf = (size_t) f * np + i;
			ShadowRay* const rays = pr.rays + 2 * ((size_t) f * np + number);
			uint32_t modes = 0;
			if (active) {
				ReservoirRecord r;
				if (kUniform) {
					const int n = pr.scene.light_count;
					const uint32_t rn_x = pr.animate ? wang_random_number((pr.noise_seed + f) * 4u) : 0u;
					uint32_t seed = get_noise_accessor(i % pr.width, i / pr.width, pr.width, rn_x);
					const int idx = (int) (get_noise_1(seed) * (float) n);
					r = ReservoirRecord{idx > n - 1 ? n - 1 : idx, 0.0f, 0.0f, seed};
					pr.records[pf] = r;
				} else {
					r = pr.records[pf];
				}
				if (r.light_index >= 0) {
					Light l;
					load_light(pr.scene, r.light_index, l);
					uint32_t seed = r.seed;
					// Contributions and rays go to memory inside.
					SampleRecord* const dst = pr.samples + pf;
					modes = psa_mis_emit<P, true>(
					    sp, peters, sd, ltc, l, light_record(pr.scene, r.light_index), seed,
					    [dst](int j, f3 c0, f3 c1) { store_contributions(dst, j, c0, c1); }, rays, poly);
					float W = P::div(r.w_sum, (float) pr.candidate_count * r.p_hat);
					if (r.p_hat == 0.0f) W = 0.0f;
					if (kUniform) W = (float) pr.scene.light_count;
					*reinterpret_cast<float2*>(reinterpret_cast<float*>(pr.samples + pf) + 12) =
					    make_float2(W, __uint_as_float(modes));
					if (numbered) pr.samples[pf].number = number;
				} else {
					const f3 zero[2][2] = {{splat(0.0f), splat(0.0f)}, {splat(0.0f), splat(0.0f)}};
					store_sample(pr.samples + pf, zero, 0.0f, kSampleNoLight);
				}
			}
			const bool t0 = (modes & 3u) == kSampleTraced, t1 = ((modes >> 2) & 3u) == kSampleTraced;
			const bool place = numbered ? active : i < np;
			if (place && !t0) store_no_ray(rays);
			if (place && !t1) store_no_ray(rays + 1);
			const uint32_t count = __popc(__ballot_sync(0xffffffffu, t0)) + __popc(__ballot_sync(0xffffffffu, t1));
			if (threadIdx.x % 32 == 0 && count) atomicAdd(&pr.counters->rays, count);
		}
	}
}

// Each warp takes 32 consecutive pixels at a time from the launch's cursor.
template <class P, bool kUniform>
__global__ void __launch_bounds__(kSampleThreads, RISLTC_SAMPLE_MIN_BLOCKS) ris_sample_kernel(const __grid_constant__ RisParams pr) {
	wait_for_previous();
	__shared__ PsaPolygon poly[kSampleThreads];
	const uint32_t np = pr.width * pr.height;
	const uint32_t chunks = (np + 31) / 32;
	const bool numbered = !kUniform && has_numbers(pr);
	for (uint32_t c = next_warp_tile(&pr.counters->sample); c < chunks; c = next_warp_tile(&pr.counters->sample))
		sample_pixel<P, kUniform>(pr, c * 32 + threadIdx.x % 32, poly[threadIdx.x], numbered);
}

// The whole estimator of pixel i (all frames of the call) where no shadow ray is
// traced: the sample phase with the contributions kept in registers, then what
// resolve_pixel does with them.
template <class P> RL_DEV void estimate_pixel(const RisParams& pr, uint32_t i, PsaPolygon& poly) {
	const uint32_t np = pr.width * pr.height;
	risltc_reservoir_t* res = pr.reservoirs ? pr.reservoirs + i : nullptr;
	f3 mean = splat(0.0f);
	if (pr.primitive && pr.primitive[i] == 0xffffffffu) {
		if (res) *res = risltc_reservoir_t{-1, 0.0f, 0.0f, 0u};
	} else {
		ShadeParams sp;  // the fields psa_mis_emit reads
		sp.scene = pr.scene;
		sp.technique = sample_polygon_ltc_cp;
		sp.mis_heuristic = pr.mis_heuristic;
		sp.mis_visibility_estimate = pr.mis_visibility_estimate;
		sp.fast_atan = pr.fast_atan;
		ShadingData sd;
		Ltc ltc;
		load_pixel<P>(pr, i, sd, ltc);
		f3 sum = splat(0.0f);
		double acc[3] = {0.0, 0.0, 0.0};
		for (uint32_t f = 0; f != pr.frame_count; ++f) {
			const ReservoirRecord r = pr.records[(size_t) f * np + i];
			f3 final_color = splat(0.0f);
			if (r.light_index >= 0) {
				Light l;
				load_light(pr.scene, r.light_index, l);
				uint32_t seed = r.seed;
				f3 own_d = splat(0.0f), own_s = splat(0.0f);
				const uint32_t modes = psa_mis_emit<P, false>(
				    sp, true, sd, ltc, l, light_record(pr.scene, r.light_index), seed,
				    [&](int j, f3 c0, f3) { (j == 0 ? own_d : own_s) = c0; }, nullptr, poly);
				f3 result = splat(0.0f);
				if ((modes & 3u) != kSampleSkip) result = add(result, own_d);
				if ((modes >> 2) != kSampleSkip) result = add(result, own_s);
				float W = P::div(r.w_sum, (float) pr.candidate_count * r.p_hat);
				if (r.p_hat == 0.0f) W = 0.0f;
				const f3 cw = scale(scale(result, P::rcp(1.0f)), W);
				final_color = add(final_color, mk3(P::div(cw.x, 1.0f), P::div(cw.y, 1.0f), P::div(cw.z, 1.0f)));
			}
			if (isnan(final_color.x) || isnan(final_color.y) || isnan(final_color.z) || isinf(final_color.x) ||
			    isinf(final_color.y) || isinf(final_color.z))
				final_color = mk3(1.0f, 0.0f, 0.8f);
			if (f == 0 && res) *res = risltc_reservoir_t{r.light_index, r.w_sum, r.p_hat, 0u};
			sum = add(sum, final_color);
			acc[0] += (double) final_color.x;
			acc[1] += (double) final_color.y;
			acc[2] += (double) final_color.z;
		}
		mean = pr.frame_count == 1 ? sum : scale(sum, 1.0f / (float) pr.frame_count);
		if (pr.accum) {
			pr.accum[3 * (size_t) i + 0] += acc[0];
			pr.accum[3 * (size_t) i + 1] += acc[1];
			pr.accum[3 * (size_t) i + 2] += acc[2];
		}
	}
	if (pr.out_rgb) {
		pr.out_rgb[3 * (size_t) i + 0] = mean.x;
		pr.out_rgb[3 * (size_t) i + 1] = mean.y;
		pr.out_rgb[3 * (size_t) i + 2] = mean.z;
	}
}

// Default calls without shadow rays.  One polygon buffer per thread, prepared
// for one space after the other, and no traversal code: 1.43 ms per 2-frame
// 1904x905 launch against 1.69 with ris_shade_kernel (two buffers, spills),
// 24.8 against 25.4 us at 256x256 (one partial wave).
template <class P>
__global__ void __launch_bounds__(kSampleThreads, RISLTC_SAMPLE_MIN_BLOCKS) ris_estimate_kernel(const __grid_constant__ RisParams pr) {
	wait_for_previous();
	__shared__ PsaPolygon poly[kSampleThreads];
	const uint32_t np = pr.width * pr.height;
	const uint32_t chunks = (np + 31) / 32;
	for_warp_tiles(&pr.counters->sample, chunks, [&](uint32_t c) {
		const uint32_t i = c * 32 + threadIdx.x % 32;
		if (i < np) estimate_pixel<P>(pr, i, poly[threadIdx.x]);
		__syncwarp();
	});
}

// Resident blocks and idle lanes per refill of the trace kernels: trace time
// per 4-frame 1080p launch with 1M occluders 3.96 ms as the compiler likes it
// (52 registers, 9 blocks), 3.78 with 10, 3.44 with 12, 4.75 with 16 (spills);
// refilling at 8, 10, 12 and 16 idle lanes 3.44, 3.37, 3.36 and 3.42.
#ifndef RISLTC_TRACE_MIN_BLOCKS
#define RISLTC_TRACE_MIN_BLOCKS 12
#endif
#ifndef RISLTC_TRACE_REFILL
#define RISLTC_TRACE_REFILL 12
#endif
// Persistent any-hit tracing of a queue of n rays.  Each lane holds one ray and advances it by one unit of
// work (a triangle test or an inner node) per iteration; whenever
// RISLTC_TRACE_REFILL or more lanes of a warp are idle they fetch the next
// rays together, so lanes do not wait for the warp's longest ray.  Queue
// has the fetch cursor (zero at launch), supplies ray k (its origin, direction and interval) and takes its outcome.
// kShared false: no cursor, each warp takes 32 rays of every gridful of them.
// (2M and 4M of a caller's rays 612 and 1,140 us, against 574 and 1,070 with
// the cursor and 700 and 1,332 with a thread per ray.)
template <class P, bool kShared, class Queue>
RL_DEV void trace_queue(const SceneView& s, const Queue& queue, uint32_t n, uint32_t* error) {
	const uint32_t lane = threadIdx.x % 32;
	const uint32_t stride = gridDim.x * blockDim.x, first = blockIdx.x * blockDim.x + threadIdx.x - lane;
	uint32_t taken = 0;
	int32_t stack[kTraceStack];
	TraceRay r;
	uint32_t k = 0;
	bool busy = false, drained = false;
	for (;;) {
		const uint32_t idle = __ballot_sync(0xffffffffu, !busy);
		if (drained && idle == 0xffffffffu) break;
		if (!drained && __popc(idle) >= RISLTC_TRACE_REFILL) {
			const int leader = __ffs(idle) - 1;
			uint32_t base = 0;
			if (kShared) {
				if ((int) lane == leader) base = atomicAdd(queue.cursor, (uint32_t) __popc(idle));
				base = __shfl_sync(0xffffffffu, base, leader);
				drained = base + (uint32_t) __popc(idle) >= n;
			} else {
				base = taken;
				taken += (uint32_t) __popc(idle);
				drained = (uint64_t) (taken / 32) * stride + first + taken % 32 >= n;
			}
			if (!busy) {
				k = base + (uint32_t) __popc(idle & ((1u << lane) - 1u));
				bool any = k < n;
				if (!kShared) {
					const uint64_t g = (uint64_t) (k / 32) * stride + first + k % 32;
					any = g < n;
					k = (uint32_t) g;
				}
				if (any) {
					f3 o, d;
					float t_min, t_max;
					queue.ray(k, o, d, t_min, t_max);
					const int st = trace_begin<P>(s, r, o, d, t_min, t_max, stack);
					if (st == kTraceContinue)
						busy = true;
					else
						queue.outcome(k, st == kTraceHit);
				}
			}
			continue;
		}
		if (busy) {
			const int st = trace_step<P>(s, r, stack, error);
			if (st != kTraceContinue) {
				queue.outcome(k, st == kTraceHit);
				busy = false;
			}
		}
	}
}

// The shading phase's rays.
struct ShadowQueue {
	const ShadowRay* rays;
	uint8_t* hits;
	uint32_t* cursor;
	RL_DEV void ray(uint32_t k, f3& o, f3& d, float& t_min, float& t_max) const {
		const float4 a = __ldg(&rays[k].origin), b = __ldg(&rays[k].dir_tmax);
		o = mk3(a.x, a.y, a.z);
		d = mk3(b.x, b.y, b.z);
		t_min = 1.0e-3f;
		t_max = b.w;
	}
	RL_DEV void outcome(uint32_t k, bool hit) const { hits[k] = hit ? 1 : 0; }
};
template <class P>
__global__ void __launch_bounds__(128, RISLTC_TRACE_MIN_BLOCKS)
shadow_trace_kernel(SceneView s, const ShadowRay* rays, uint32_t count, uint32_t* cursor, uint8_t* hits, uint32_t* error) {
	allow_next();
	trace_queue<P, true>(s, ShadowQueue{rays, hits, cursor}, count, error);
}

// The same loop over a source of rays that deals them out itself: deal(idle,
// drained) is called by whole warps with the idle lanes' mask, true for a lane
// that got a ray, drained when there are no more.  The source gives the lane's
// ray and its scene and takes its outcome.
template <class P, class Source> RL_DEV void trace_dealt(Source& source, uint32_t* error) {
	int32_t stack[kTraceStack];
	TraceRay r;
	bool busy = false, drained = false;
	for (;;) {
		const uint32_t idle = __ballot_sync(0xffffffffu, !busy);
		if (drained && idle == 0xffffffffu) break;
		if (!drained && __popc(idle) >= RISLTC_TRACE_REFILL) {
			if (source.deal(idle, drained)) {
				f3 o, d;
				float t_min, t_max;
				source.ray(o, d, t_min, t_max);
				const int st = trace_begin<P>(source.scene(), r, o, d, t_min, t_max, stack);
				if (st == kTraceContinue)
					busy = true;
				else
					source.outcome(st == kTraceHit);
			}
			continue;
		}
		if (busy) {
			const int st = trace_step<P>(source.scene(), r, stack, error);
			if (st != kTraceContinue) {
				source.outcome(st == kTraceHit);
				busy = false;
			}
		}
	}
}

// Places of a queue that a warp has claimed and not dealt out yet, from claimed.x
// to claimed.y (in shared memory, a slot per warp: two registers made the batch
// kernel spill).  A claim takes what the idle lanes want or, while more remain,
// a share of the remaining places, 2^-shift: a cursor answers one claim after
// another, 0.7 ns each, and places without a ray are done faster than that.
RL_DEV bool deal_places(uint32_t idle, bool& drained, uint2& claimed, uint32_t count, int shift, uint32_t& place, uint32_t* cursor) {
	const uint32_t lane = threadIdx.x % 32, n = (uint32_t) __popc(idle);
	const uint32_t rank = (uint32_t) __popc(idle & ((1u << lane) - 1u));
	uint32_t next = claimed.x, end = claimed.y;
	const uint32_t left = end - next;
	uint32_t at = next + rank;
	next += n;
	if (left < n) {
		const uint32_t size = max(n - left, (count - min(end, count)) >> shift);
		uint32_t base = 0;
		if (lane == 0) base = atomicAdd(cursor, size);
		base = __shfl_sync(0xffffffffu, base, 0);
		if (rank >= left) at = base + rank - left;
		next = base + n - left;
		end = base + size;
	}
	__syncwarp();
	if (lane == 0) claimed = make_uint2(next, end);
	__syncwarp();
	drained = next >= count;
	place = at;
	return (idle >> lane & 1u) && at < count;
}

// The rays of a call with many places, claimed by shares.
struct FrameRays {
	const SceneView& s;
	const ShadowRay* rays;
	uint8_t* hits;
	uint32_t* cursor;
	uint32_t covered, pixels, frames;
	int shift;
	uint2& claimed;
	uint32_t place;  // the lane's

	RL_DEV bool deal(uint32_t idle, bool& drained) {
		uint32_t g;
		if (!deal_places(idle, drained, claimed, 2u * covered * frames, shift, g, cursor)) return false;
		place = queue_place(g, covered, pixels);
		return true;
	}
	RL_DEV const SceneView& scene() const { return s; }
	RL_DEV void ray(f3& o, f3& d, float& t_min, float& t_max) const {
		const float4 a = __ldg(&rays[place].origin), b = __ldg(&rays[place].dir_tmax);
		o = mk3(a.x, a.y, a.z);
		d = mk3(b.x, b.y, b.z);
		t_min = 1.0e-3f;
		t_max = b.w;
	}
	RL_DEV void outcome(bool hit) const { hits[place] = hit ? 1 : 0; }
};
template <class P>
__global__ void __launch_bounds__(128, RISLTC_TRACE_MIN_BLOCKS)
shadow_trace_shares_kernel(SceneView s, const ShadowRay* rays, uint32_t pixels, uint32_t frames, int shift,
                           LaunchCounters* counters, uint8_t* hits, uint32_t* error) {
	__shared__ uint2 claimed[4];
	claimed[threadIdx.x / 32] = make_uint2(0u, 0u);
	__syncwarp();
	allow_next();
	FrameRays source{s, rays, hits, &counters->fetch, queue_covered(counters, pixels), pixels, frames, shift,
	                 claimed[threadIdx.x / 32], 0u};
	trace_dealt<P>(source, error);
}
// The shift: at least 15 (for the 7,296 warps of a full grid a claim is at most
// two ninths of a warp's even share of what remains), and no claim of more than
// 256 places, which warps that come to them last would be left alone with.
inline int claim_shift(uint32_t count) {
	int shift = 15;
	while ((count >> shift) > 256u) ++shift;
	return shift;
}
// Places per lane of a full grid from which queues with background are numbered
// and claims made by shares.  Above: 4-frame 1080p calls with 16,384 lights take
// 14.60 ms without background (14.61 with single claims and every pixel's places
// kept), 1.48 with 95% of it above a horizon (2.15; 2.09 when the rays were
// compacted and grouped by light, which all else paid for), 0.36 with nothing
// else (0.78; 0.42); one frame with 1,024 lights 3.78, 0.53 and 0.18 ms (3.78,
// 0.60, 0.26; 5.36, 0.64, 0.19).  Below, calls of 3 frames of 961x541 with any
// background but all lose 1% or less to the empty places.
constexpr uint32_t kSharesPerLane = 16;

// Whether a 32-bit cursor can deal out `rays` to `threads` threads: after the
// last ray each warp may add up to 32 once more, and a cursor that wrapped there
// would deal the first rays out again, and again after them.
constexpr bool cursor_holds(uint32_t rays, uint32_t threads) { return rays <= 0xffffffffu - threads; }

// A caller's rays (risltc_trace_shadow).
struct CallerQueue {
	const float4* rays;
	uint32_t* hits;
	uint32_t* cursor;
	RL_DEV void ray(uint32_t k, f3& o, f3& d, float& t_min, float& t_max) const {
		const float4 a = rays[2 * (size_t) k], b = rays[2 * (size_t) k + 1];
		o = mk3(a.x, a.y, a.z);
		d = mk3(b.x, b.y, b.z);
		t_min = a.w;
		t_max = b.w;
	}
	RL_DEV void outcome(uint32_t k, bool hit) const { hits[k] = hit ? 1u : 0u; }
};
template <class P, bool kShared>
__global__ void __launch_bounds__(128, RISLTC_TRACE_MIN_BLOCKS) trace_shadow_queue_kernel(SceneView s, const float4* rays, uint32_t count,
                                                                 uint32_t* hits, uint32_t* cursor, uint32_t* error) {
	trace_queue<P, kShared>(s, CallerQueue{rays, hits, cursor}, count, error);
}

// The resolve phase of pixel i (all frames of the call); i may be past the
// frame (nothing is done then).
template <class P> RL_DEV void resolve_pixel(const RisParams& pr, uint32_t i) {
	const uint32_t np = pr.width * pr.height;
	if (i >= np) return;
	{
		risltc_reservoir_t* res = pr.reservoirs ? pr.reservoirs + i : nullptr;
		if (pr.primitive && pr.primitive[i] == 0xffffffffu) {
			if (res) *res = risltc_reservoir_t{-1, 0.0f, 0.0f, 0u};
			if (pr.out_rgb) {
				pr.out_rgb[3 * (size_t) i + 0] = 0.0f;
				pr.out_rgb[3 * (size_t) i + 1] = 0.0f;
				pr.out_rgb[3 * (size_t) i + 2] = 0.0f;
			}
			return;
		}
		const bool numbered = has_numbers(pr);
		f3 sum = splat(0.0f);
		double acc[3] = {0.0, 0.0, 0.0};
		for (uint32_t f = 0; f != pr.frame_count; ++f) {
			const size_t pf = (size_t) f * np + i;
			const float4* q = reinterpret_cast<const float4*>(pr.samples + pf);
			const float4 q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3];
			const uint32_t flags = __float_as_uint(q3.y);
			f3 final_color = splat(0.0f);
			if (!(flags & kSampleNoLight)) {
				const f3 c[2][2] = {{mk3(q0.x, q0.y, q0.z), mk3(q0.w, q1.x, q1.y)},
				                    {mk3(q1.z, q1.w, q2.x), mk3(q2.y, q2.z, q2.w)}};
				f3 result = splat(0.0f);
#pragma unroll
				for (int j = 0; j != 2; ++j) {
					const uint32_t mode = (flags >> (2 * j)) & 3u;
					if (mode == kSampleSkip) continue;
					const bool occluded = mode == kSampleTraced && pr.hits[2 * ((size_t) f * np + (numbered ? __float_as_uint(q3.z) : i)) + j] != 0;
					result = add(result, occluded ? c[j][1] : c[j][0]);
				}
				const f3 color = scale(result, P::rcp(1.0f));
				const f3 cw = scale(color, q3.x);
				final_color = add(final_color, mk3(P::div(cw.x, 1.0f), P::div(cw.y, 1.0f), P::div(cw.z, 1.0f)));
			}
			const bool finite = !(isnan(final_color.x) || isnan(final_color.y) || isnan(final_color.z) ||
			                      isinf(final_color.x) || isinf(final_color.y) || isinf(final_color.z));
			if (f == 0 && pr.train_shaded && pr.train_stride && i % pr.train_stride == pr.train_phase)
				pr.train_shaded[i] =
				    finite ? 0.2126f * final_color.x + 0.7152f * final_color.y + 0.0722f * final_color.z : 0.0f;
			if (!finite) final_color = mk3(1.0f, 0.0f, 0.8f);
			if (f == 0 && res) {
				const ReservoirRecord r = pr.records[pf];
				*res = risltc_reservoir_t{r.light_index, r.w_sum, r.p_hat, 0u};
			}
			sum = add(sum, final_color);
			acc[0] += (double) final_color.x;
			acc[1] += (double) final_color.y;
			acc[2] += (double) final_color.z;
		}
		if (pr.out_rgb) {
			f3 mean = pr.frame_count == 1 ? sum : scale(sum, 1.0f / (float) pr.frame_count);
			pr.out_rgb[3 * (size_t) i + 0] = mean.x;
			pr.out_rgb[3 * (size_t) i + 1] = mean.y;
			pr.out_rgb[3 * (size_t) i + 2] = mean.z;
		}
		if (pr.accum) {
			pr.accum[3 * (size_t) i + 0] += acc[0];
			pr.accum[3 * (size_t) i + 1] += acc[1];
			pr.accum[3 * (size_t) i + 2] += acc[2];
		}
	}
}

template <class P> __global__ void __launch_bounds__(128) ris_resolve_kernel(const __grid_constant__ RisParams pr) {
	wait_for_previous();
	const uint32_t np = pr.width * pr.height;
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x)
		resolve_pixel<P>(pr, i);
}

}  // namespace risltc
