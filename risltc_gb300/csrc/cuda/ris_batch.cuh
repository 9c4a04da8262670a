// ris_batch.cuh - the wavefront pipeline of the default configuration run
// over a batch of frames (risltc_shade_batch) with one launch per phase: the
// candidate, sample, trace and resolve kernels each take their work units
// (warp tiles, pixels, rays) from the concatenation of all items' units, so a
// batch of small and large frames fills the GPU in four launches instead of
// four per item.
//
// Every unit runs the single-frame kernels' body (binned_tile, sample_pixel,
// the trace loop, resolve_pixel) with its item's parameters, so each item's
// results are bit-identical to its own risltc_shade call.  The items'
// parameters travel in kernel parameter space (RisBatch, about 2.2 KB for 8
// items) and are captured by value into a CUDA graph.
#pragma once
#include "ris_binned.cuh"
#include "ris_wavefront.cuh"

namespace risltc {

// Items per whole-batch launch; risltc_shade_batch runs larger batches in
// groups of this many beside each other.  Batches of 9, 12, 16, 20 and 33 small
// frames (64 to 200 pixels wide, 5,000 occluders) take 197, 218, 271, 343 and
// 544 us; groups of 16 one after the other 206, 222, 262, 386 and 614, groups of
// 8 one after the other 318, 316, 342, 460 and 788.  Large frames (256 to 1,400
// wide): 16 of them 5.01, 4.92 and 5.02 ms, 33 of them 9.95, 9.99 and 10.16.
constexpr int kBatchItems = 8;

struct RisBatch {
	uint32_t count;
	// Prefix sums over the items of their candidate tiles (kPixels pixels
	// each, for the tile shape of the launch) and of their pixels, each item's
	// rounded up to whole warps of 32, and of their queue places (two per
	// pixel-frame).
	uint32_t tile_begin[kBatchItems + 1];
	uint32_t pixel_begin[kBatchItems + 1];
	uint32_t ray_begin[kBatchItems + 1];
	// The candidate kernel's per-warp p_hat slots (for the launch's grid).
	float* p_hat_scratch;
	// The batch's cursors over all items' units; the items' ray counts are in
	// their own counters.  Zeroed before the launches, as the items' are.
	LaunchCounters* counters;
	RisParams item[kBatchItems];
};

// The item whose units begin[k] .. begin[k + 1] - 1 hold unit u (begin has
// count + 1 entries, u < begin[count]).
RL_DEV uint32_t batch_item(const uint32_t* begin, uint32_t count, uint32_t u) {
	uint32_t lo = 0, hi = count - 1;
	while (lo < hi) {
		const uint32_t mid = (lo + hi + 1) >> 1;
		if (begin[mid] <= u)
			lo = mid;
		else
			hi = mid - 1;
	}
	return lo;
}

template <class P, int kPixels, int kChunk>
__global__ void __launch_bounds__(32 * kBinnedWarps, BinnedMinBlocks<P>::value)
ris_candidates_batch_kernel(const __grid_constant__ RisBatch b) {
	extern __shared__ __align__(16) unsigned char smem_raw[];
	using Tile = WarpTile<BinnedSuper<P>::value, kPixels, kChunk>;
	Tile& tile = reinterpret_cast<Tile*>(smem_raw)[threadIdx.x / 32];
	float* const phat = b.p_hat_scratch + (size_t) (blockIdx.x * kBinnedWarps + threadIdx.x / 32) * kPHatSlot;
	const uint32_t tiles = b.tile_begin[b.count];
	for (uint32_t u = next_warp_tile(&b.counters->tile); u < tiles; u = next_warp_tile(&b.counters->tile)) {
		const uint32_t k = batch_item(b.tile_begin, b.count, u);
		binned_tile<P, kPixels, kChunk>(b.item[k], tile, phat, u - b.tile_begin[k]);
	}
}

template <class P, int kPixels, int kChunk>
cudaError_t launch_candidates_batch(const RisBatch& b, cudaStream_t stream, int grid_cap) {
	static std::atomic<uint64_t> configured{0};
	static std::atomic<int> resident[64];
	int device = 0;
	const cudaError_t e = configure_candidate_kernel(ris_candidates_batch_kernel<P, kPixels, kChunk>,
	                                                 binned_smem_bytes<P, kPixels, kChunk>(), configured, resident, device);
	if (e != cudaSuccess) return e;
	const size_t blocks = ((size_t) b.tile_begin[b.count] + kBinnedWarps - 1) / kBinnedWarps;
	const int grid = (int) std::max<size_t>(
	    1, std::min<size_t>(blocks, (size_t) std::min(grid_cap, resident[device & 63].load())));
	ris_candidates_batch_kernel<P, kPixels, kChunk>
	    <<<grid, 32 * kBinnedWarps, binned_smem_bytes<P, kPixels, kChunk>(), stream>>>(b);
	return cudaGetLastError();
}

template <class P>
__global__ void __launch_bounds__(kSampleThreads, RISLTC_SAMPLE_MIN_BLOCKS) ris_sample_batch_kernel(const __grid_constant__ RisBatch b) {
	__shared__ PsaPolygon poly[kSampleThreads];
	const uint32_t chunks = b.pixel_begin[b.count] / 32;
	for (uint32_t c = next_warp_tile(&b.counters->sample); c < chunks; c = next_warp_tile(&b.counters->sample)) {
		const uint32_t u = c * 32 + threadIdx.x % 32, k = batch_item(b.pixel_begin, b.count, c * 32);
		sample_pixel<P, false>(b.item[k], u - b.pixel_begin[k], poly[threadIdx.x], has_numbers(b.item[k]));
	}
}

// Persistent any-hit tracing of all items' queues as one queue (the items'
// queues one after another), with the lane refill of shadow_trace_kernel;
// each lane traverses its ray's item's BVH and writes its item's outcome.
template <class P>
__global__ void __launch_bounds__(128, RISLTC_TRACE_MIN_BLOCKS) shadow_trace_batch_kernel(const __grid_constant__ RisBatch b) {
	const uint32_t n = b.ray_begin[b.count];
	const uint32_t lane = threadIdx.x % 32;
	uint32_t* const error = b.item[0].error;
	int32_t stack[kTraceStack];
	TraceRay r;
	SceneView s = {};
	uint8_t* hits = nullptr;
	uint32_t slot = 0;
	bool busy = false, drained = false;
	for (;;) {
		const uint32_t idle = __ballot_sync(0xffffffffu, !busy);
		if (drained && idle == 0xffffffffu) break;
		if (!drained && __popc(idle) >= RISLTC_TRACE_REFILL) {
			const int leader = __ffs(idle) - 1;
			uint32_t base = 0;
			if ((int) lane == leader) base = atomicAdd(&b.counters->fetch, (uint32_t) __popc(idle));
			base = __shfl_sync(0xffffffffu, base, leader);
			drained = base + (uint32_t) __popc(idle) >= n;
			if (!busy) {
				const uint32_t g = base + (uint32_t) __popc(idle & ((1u << lane) - 1u));
				if (g < n) {
					const uint32_t k = batch_item(b.ray_begin, b.count, g);
					const RisParams& pr = b.item[k];
					s.pairs = pr.scene.pairs;
					s.triangles = pr.scene.triangles;
					s.triangle_count = pr.scene.triangle_count;
					hits = pr.hits;
					slot = g - b.ray_begin[k];
					const ShadowRay* ray = pr.rays + slot;
					const float4 a = __ldg(&ray->origin), d = __ldg(&ray->dir_tmax);
					const int st = trace_begin<P>(s, r, mk3(a.x, a.y, a.z), mk3(d.x, d.y, d.z), 1.0e-3f, d.w, stack);
					if (st == kTraceContinue)
						busy = true;
					else
						hits[slot] = st == kTraceHit ? 1 : 0;
				}
			}
			continue;
		}
		if (busy) {
			const int st = trace_step<P>(s, r, stack, error);
			if (st != kTraceContinue) {
				hits[slot] = st == kTraceHit ? 1 : 0;
				busy = false;
			}
		}
	}
}

// The same for many places, claimed by shares, of the items' covered pixels.
struct BatchRays {
	const RisBatch& b;
	const uint32_t* begin;  // prefix sums of the items' rays
	int shift;
	uint2& claimed;
	SceneView s;            // of the lane's ray: the fields that the traversal reads,
	uint8_t* hit;           // its outcome's place
	const ShadowRay* rays;  // and its own

	RL_DEV bool deal(uint32_t idle, bool& drained) {
		uint32_t g;
		if (!deal_places(idle, drained, claimed, begin[b.count], shift, g, &b.counters->fetch)) return false;
		const uint32_t k = batch_item(begin, b.count, g);
		const RisParams& pr = b.item[k];
		s.pairs = pr.scene.pairs;
		s.triangles = pr.scene.triangles;
		s.triangle_count = pr.scene.triangle_count;
		const uint32_t n = begin[k + 1] - begin[k], pixels = pr.width * pr.height;
		g -= begin[k];
		// (n is 2 * covered * frames.)
		if (n != b.ray_begin[k + 1] - b.ray_begin[k]) g = queue_place(g, n / (2u * pr.frame_count), pixels);
		hit = pr.hits + g;
		rays = pr.rays + g;
		return true;
	}
	RL_DEV const SceneView& scene() const { return s; }
	RL_DEV void ray(f3& o, f3& d, float& t_min, float& t_max) const {
		const float4 a = __ldg(&rays->origin), r = __ldg(&rays->dir_tmax);
		o = mk3(a.x, a.y, a.z);
		d = mk3(r.x, r.y, r.z);
		t_min = 1.0e-3f;
		t_max = r.w;
	}
	RL_DEV void outcome(bool occluded) const { *hit = occluded ? 1 : 0; }
};
template <class P>
__global__ void __launch_bounds__(128, RISLTC_TRACE_MIN_BLOCKS)
shadow_trace_batch_shares_kernel(const __grid_constant__ RisBatch b, int shift) {
	__shared__ uint2 claimed[4];
	__shared__ uint32_t begin[kBatchItems + 1];
	claimed[threadIdx.x / 32] = make_uint2(0u, 0u);
	if (threadIdx.x <= b.count) {
		uint32_t sum = 0;
		for (uint32_t k = 0; k != threadIdx.x; ++k) {
			const RisParams& pr = b.item[k];
			sum += 2u * queue_covered(pr.counters, pr.width * pr.height) * pr.frame_count;
		}
		begin[threadIdx.x] = sum;
	}
	__syncthreads();
	BatchRays source{b, begin, shift, claimed[threadIdx.x / 32], SceneView{}, nullptr, nullptr};
	trace_dealt<P>(source, b.item[0].error);
}

template <class P> __global__ void __launch_bounds__(128) ris_resolve_batch_kernel(const __grid_constant__ RisBatch b) {
	const uint32_t total = b.pixel_begin[b.count];
	for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < total; u += gridDim.x * blockDim.x) {
		const uint32_t k = batch_item(b.pixel_begin, b.count, u);
		resolve_pixel<P>(b.item[k], u - b.pixel_begin[k]);
	}
}

// Launchers (shade_exact.cu; the candidate kernel's tile shapes as in the
// single-frame path: 32 x 8 there, the others in candidate_tiles.cu).
cudaError_t launch_candidates_batch_exact(const RisBatch& b, cudaStream_t stream, int grid_cap, int tile);
cudaError_t launch_candidates_batch_fast(const RisBatch& b, cudaStream_t stream, int grid_cap, int tile);
cudaError_t launch_candidates_batch_tile_exact(const RisBatch& b, cudaStream_t stream, int grid_cap, int tile);
cudaError_t launch_candidates_batch_tile_fast(const RisBatch& b, cudaStream_t stream, int grid_cap, int tile);
// Sample, trace and resolve kernels of the batch, with the given grids.
cudaError_t launch_batch_estimator(const RisBatch& b, cudaStream_t stream, int pixel_grid, int ray_grid);

}  // namespace risltc
