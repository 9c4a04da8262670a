// Instantiations compiled with --fmad=false and IEEE division and square
// root: everything that must match the CPU restatement bit for bit, plus the
// fused kernel's fast-candidate variant (its candidate loop uses hardware
// reciprocal square root; its final shading stays exact).
#include "ris_batch.cuh"

namespace risltc {
cudaError_t launch_shade(const ShadeParams& p, cudaStream_t stream, int grid, cudaEvent_t* events, bool fast) {
	if (events) cudaEventRecord(events[0], stream);
	if (fast)
		shade_kernel<FastNumerics, ExactNumerics><<<grid, kShadeThreads, 0, stream>>>(p);
	else
		shade_kernel<ExactNumerics, ExactNumerics><<<grid, kShadeThreads, 0, stream>>>(p);
	cudaError_t e = cudaGetLastError();
	if (events)
		for (int k = 1; k != RISLTC_PROFILE_PHASES + 1; ++k) cudaEventRecord(events[k], stream);
	return e;
}
cudaError_t launch_candidates_exact(const RisParams& p, cudaStream_t stream, int grid_cap, int tile) {
	if (tile == risltc_tile_32x8) return launch_candidates_binned<ExactNumerics, 32, 8>(p, stream, grid_cap);
	if (tile == risltc_tile_per_pixel) {
		ris_candidates_kernel<ExactNumerics>
		    <<<grid_for_pixels((size_t) p.width * p.height, grid_cap), 128, 0, stream>>>(p);
		return cudaGetLastError();
	}
	return launch_candidates_tile_exact(p, stream, grid_cap, tile);
}
cudaError_t launch_ris_shade(const RisParams& p, cudaStream_t stream, int grid) {
	ris_shade_kernel<ExactNumerics><<<grid, kShadeThreads, 0, stream>>>(p);
	return cudaGetLastError();
}
cudaError_t launch_proposal(const ProposalParams& p, cudaStream_t stream, int grid) {
	proposal_kernel<<<grid, 32 * kProposalWarps, proposal_smem_bytes(p.clusters.count), stream>>>(p);
	return cudaGetLastError();
}
cudaError_t launch_ris_sample(const RisParams& p, cudaStream_t stream, int grid) {
	if (p.uniform_light)
		return launch_behind(p.overlap != 0, ris_sample_kernel<ExactNumerics, true>, grid, kSampleThreads, stream, p);
	return launch_behind(p.overlap != 0, ris_sample_kernel<ExactNumerics, false>, grid, kSampleThreads, stream, p);
}
cudaError_t launch_ris_estimate(const RisParams& p, cudaStream_t stream, int grid) {
	return launch_behind(p.overlap != 0, ris_estimate_kernel<ExactNumerics>, grid, kSampleThreads, stream, p);
}
cudaError_t launch_shadow_trace(const RisParams& p, cudaStream_t stream, int grid) {
	const uint32_t count = 2u * p.width * p.height * p.frame_count;
	// Never early: its blocks would gather on the SMs that drain first (a 349x168
	// frame took 157 instead of 144 us).
	if (p.compact)
		shadow_trace_shares_kernel<ExactNumerics>
		    <<<grid, 128, 0, stream>>>(p.scene, p.rays, p.width * p.height, p.frame_count, claim_shift(count), p.counters,
		                               p.hits, p.error);
	else
		shadow_trace_kernel<ExactNumerics>
		    <<<grid, 128, 0, stream>>>(p.scene, p.rays, count, &p.counters->fetch, p.hits, p.error);
	return cudaGetLastError();
}
cudaError_t launch_ris_resolve(const RisParams& p, cudaStream_t stream, int grid) {
	return launch_behind(p.overlap != 0, ris_resolve_kernel<ExactNumerics>, grid, 128, stream, p);
}
cudaError_t launch_candidates_batch_exact(const RisBatch& b, cudaStream_t stream, int grid_cap, int tile) {
	if (tile == risltc_tile_32x8) return launch_candidates_batch<ExactNumerics, 32, 8>(b, stream, grid_cap);
	return launch_candidates_batch_tile_exact(b, stream, grid_cap, tile);
}
cudaError_t launch_batch_estimator(const RisBatch& b, cudaStream_t stream, int pixel_grid, int ray_grid) {
	ris_sample_batch_kernel<ExactNumerics><<<pixel_grid, kSampleThreads, 0, stream>>>(b);
	cudaError_t e = cudaGetLastError();
	if (e != cudaSuccess) return e;
	if (b.item[0].compact)
		shadow_trace_batch_shares_kernel<ExactNumerics><<<ray_grid, 128, 0, stream>>>(b, claim_shift(b.ray_begin[b.count]));
	else
		shadow_trace_batch_kernel<ExactNumerics><<<ray_grid, 128, 0, stream>>>(b);
	if ((e = cudaGetLastError()) != cudaSuccess) return e;
	ris_resolve_batch_kernel<ExactNumerics><<<pixel_grid, 128, 0, stream>>>(b);
	return cudaGetLastError();
}
// One thread per ray while all of them are resident at once (blocks of 128),
// the persistent queue beyond that, whose cursor (if any that holds the count)
// is zeroed first: 2M rays against 200k occluders took 831 us with a thread per ray, 667 with the
// queue when it was brought in and 576 with the present traversal.
cudaError_t launch_trace_exact(const SceneView& s, const float4* rays, uint32_t count, uint32_t* hits, uint32_t* error,
                               uint32_t* cursor, cudaStream_t stream, int resident) {
	const int grid = (int) (((size_t) count + 127) / 128);
	if (grid <= resident) {
		trace_shadow_kernel<ExactNumerics><<<grid, 128, 0, stream>>>(s, rays, count, hits, error);
		return cudaGetLastError();
	}
	if (!cursor || !cursor_holds(count, (uint32_t) resident * 128)) {
		trace_shadow_queue_kernel<ExactNumerics, false><<<resident, 128, 0, stream>>>(s, rays, count, hits, cursor, error);
		return cudaGetLastError();
	}
	const cudaError_t e = cudaMemsetAsync(cursor, 0, sizeof(uint32_t), stream);
	if (e != cudaSuccess) return e;
	trace_shadow_queue_kernel<ExactNumerics, true><<<resident, 128, 0, stream>>>(s, rays, count, hits, cursor, error);
	return cudaGetLastError();
}
}  // namespace risltc
