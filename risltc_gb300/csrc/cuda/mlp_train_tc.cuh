// mlp_train_tc.cuh - online training of the proposal MLP on the tcgen05
// tensor cores (up to 256 clusters): forward pass, softmax cross-entropy
// gradient, the backward products and the weight gradients of a training
// step, with BF16 operands and FP32 accumulators.
//
// One CTA of 16 warps per SM takes tiles of 128 training pixels, four threads to
// a pixel, each with a quarter of every row's columns.  All operands live in shared memory in the K-major 8x8 core-matrix layout of
// the forward pass ([pixel][feature] for activations and gradients,
// [out][in] for weights).  The products that contract over the pixels (the
// weight gradients) and over a weight matrix's rows (the input gradients)
// read the same bytes through MN-major descriptors, so nothing is stored
// twice.  Per tile:
//   D1 = E W1^T, H1 = ReLU(D1 + b1); D2 = H1 W2^T, H2 = ReLU(D2 + b2);
//   logits in chunks of 128 clusters, BF16 in registers, softmax per pixel;
//   DZ = (q - T) / B as in the CUDA-core kernel (each thread subtracts its
//   own columns' part of the target T);
//   dh2 = DZ W3 and dW3 += DZ^T [H2 | 1]; DZ2 = dh2 * [H2 > 0];
//   dh1 = DZ2 W2 and dW2 += DZ2^T [H1 | 1]; DZ1 = dh1 * [H1 > 0];
//   dW1 += DZ1^T E (feature 130 of E is 1, so its column is db1).
// The weight gradients accumulate in tensor memory over all tiles of the
// CTA and are added to the FP32 gradient vector once at the end.  Tensor
// memory (512 columns): 0..127 the per-tile products, 128..287 dW3 (80
// columns per 128-cluster chunk: 64 weights, the bias, 15 zeros), 288..367
// dW2, 368..511 dW1.  The hidden layers' M = 64 weight-gradient products run
// at M = 128; their upper 64 rows read the following bytes of shared memory
// and are discarded.
//
// What bounds it: a tile is a chain (products, epilogues, softmax) with nothing
// else on the SM to run meanwhile, 37 thousand cycles long for 256 clusters and
// 32 candidates: about 8 of them products, 10 the logits and their two passes of
// exponentials, 7 the candidates.  So the chain's links are split over 16 warps,
// and the next tile's candidates and inputs are fetched behind the backward
// products.  One step of 129,600 pixels takes 145 us; with four warps, a thread
// per pixel, 207 us; of that the candidates, which each thread read for itself,
// were the largest part, and with more warps alone they grew (225 us).
#pragma once
#include "mlp_tc.cuh"

namespace risltc {

constexpr int kTtMaxClusters = 256;
constexpr int kTtHiddenCols = 80;                    // stored hidden columns: 64 values, 1.0, 15 zeros
constexpr int kTtOnesFeature = kMlpInputs * 13;     // feature 130 (a padding feature, zero weight)
constexpr int kTtSplit = 4;  // threads per row of a tile, each with a part of its columns
constexpr int kTtThreads = kTtSplit * kTcRows;
constexpr uint32_t kTtColumns = 512;
constexpr uint32_t kTtGrad3 = 128, kTtGrad2 = 288, kTtGrad1 = 368;
// Shared memory (bytes).
constexpr uint32_t kTtW1 = 0;
constexpr uint32_t kTtW2 = kTtW1 + kMlpHidden * kMlpFeatures * 2;
constexpr uint32_t kTtW3 = kTtW2 + kMlpHidden * kMlpHidden * 2;
constexpr uint32_t kTtE = kTtW3 + kTtMaxClusters * kMlpHidden * 2;
constexpr uint32_t kTtH1 = kTtE + kTcRows * kMlpFeatures * 2;
constexpr uint32_t kTtH2 = kTtH1 + kTcRows * kTtHiddenCols * 2;
constexpr uint32_t kTtDz = kTtH2 + kTcRows * kTtHiddenCols * 2;
constexpr uint32_t kTtD = kTtDz + kTcRows * kTtMaxClusters * 2;  // DZ2, then DZ1
constexpr uint32_t kTtBias = kTtD + kTcRows * kMlpHidden * 2;    // b1, b2, b3 (FP32)
constexpr uint32_t kTtBar = kTtBias + (2 * kMlpHidden + kTtMaxClusters) * 4;
constexpr uint32_t kTtSlot = kTtBar + 16;
// A tile's first kTtHeld candidates per row: their weights in D, which is free
// until the backward pass, their clusters here; the rows' maxima and sums by
// parts of the columns.
constexpr int kTtHeld = 32;
constexpr uint32_t kTtCluster = (kTtSlot + 8 + 15) / 16 * 16;
constexpr uint32_t kTtSum = kTtCluster + kTtHeld * kTcRows * 2;
constexpr uint32_t kTtMax = kTtSum + kTtSplit * kTcRows * 4;
constexpr uint32_t kTtSmemBytes = kTtMax + kTtSplit * kTcRows * 2;
// The M = 128 reads of DZ2/DZ1 reach 1 KB past their buffer (into the biases).
static_assert(kTtBias - kTtD + (2 * kMlpHidden + kTtMaxClusters) * 4 >= 14 * 1024 + 16 * 128 + 1024 + 128,
              "the discarded rows of the hidden weight-gradient products stay in shared memory");
static_assert(kTtHeld * kTcRows * 4 <= kTcRows * kMlpHidden * 2, "a tile's candidate weights fit in D");
static_assert(kTtMaxClusters <= 65535 && kTtSum % 4 == 0 && kTtD % 16 == 0, "clusters in 16 bits");
static_assert(kTtSmemBytes <= 232448, "fits one CTA per SM");

// Shared-memory descriptor (no swizzle, version 1): `leading` is the byte
// distance between core matrices along K, `stride` along M or N, for both
// K-major and MN-major operands.
RL_DEV uint64_t tc_descriptor_mn(uint32_t addr, uint32_t leading, uint32_t stride) {
	return (uint64_t) ((addr & 0x3FFFFu) >> 4) | ((uint64_t) (leading >> 4) << 16) | ((uint64_t) (stride >> 4) << 32) |
	       (1ull << 46);
}
constexpr uint32_t kTcAMajorMN = 1u << 15, kTcBMajorMN = 1u << 16;

// 16 consecutive FP32 columns of this thread's tensor-memory lane.
RL_DEV void tc_load16(uint32_t taddr, uint32_t (&v)[16]) {
	asm volatile(
	    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
	    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
	      "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
	    : "r"(taddr));
}

RL_DEV float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
RL_DEV float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// The cluster of a candidate, kNoCluster where it is no target.
constexpr uint32_t kNoCluster = 0xffffffffu;
RL_DEV uint32_t candidate_cluster(const MlpTrainParams& pr, int light, float w) {
	return w > 0.0f && (uint32_t) light < pr.light_count ? pr.light_cluster[light] : kNoCluster;
}

// Where row `row`'s candidate c is staged: a row's weights in eight 16-byte
// words and its clusters in four, permuted so that eight consecutive rows' words
// of one index fall in distinct banks.
RL_DEV int staged_weight(int c, int row) { return row * kTtHeld + (((c >> 2) ^ (row & 7)) << 2) + (c & 3); }
RL_DEV int staged_cluster(int c, int row) { return row * kTtHeld + (((c >> 3) ^ (row >> 1 & 3)) << 3) + (c & 7); }

// Loads that stay where they are written: the compiler moved plain ones down to
// their use, behind the waits that are to hide them.
RL_DEV uint32_t load_here(const void* p) {
	uint32_t v;
	asm volatile("ld.global.nc.b32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
	return v;
}
RL_DEV uint2 load_pair_here(const void* p) {  // 8-byte aligned
	uint2 v;
	asm volatile("ld.global.nc.v2.b32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
	return v;
}

// The first kTtHeld candidates of kRows rows of a tile on their way to its
// stage, by one warp: consecutive lanes read consecutive candidates, and all of
// a lane's are in flight together.  (A thread reading its own row's touched a
// line per lane and load and waited for memory several times: 20 of a tile's 52
// thousand cycles.)
template <int kRows> struct CandidateFetch {
	static constexpr int kBatch = kRows * kTtHeld / 32;
	static_assert(kRows * kTtHeld <= 256 && kTtHeld <= 32, "row(): exact for fewer than 256 candidates of at most 32 per row");
	int first, m;      // the first row, candidates per row
	uint32_t inv_m;
	int light[kBatch];  // -1: no target
	float weight[kBatch];
	uint32_t cluster[kBatch];

	RL_DEV CandidateFetch(int first_row, int count)
	    : first(first_row), m(min(count, kTtHeld)), inv_m(65536u / (uint32_t) m + 1u) {}
	RL_DEV uint32_t index(int k) const { return threadIdx.x % 32 + 32 * k; }
	RL_DEV bool any(int k) const { return index(k) < (uint32_t) (kRows * m); }
	RL_DEV int row(int k) const { return (int) (index(k) * inv_m >> 16); }  // of the kRows rows
	RL_DEV int candidate(int k) const { return (int) index(k) - row(k) * m; }

	RL_DEV void load_lights(const MlpTrainParams& pr, uint32_t j0, uint32_t n_train) {  // the tile at training pixel j0
		const bool wide = (reinterpret_cast<uintptr_t>(pr.candidates) & 7) == 0;  // else 4-byte aligned
#pragma unroll
		for (int k = 0; k != kBatch; ++k) {
			const uint32_t j = j0 + (uint32_t) (first + row(k));
			light[k] = -1;
			weight[k] = 0.0f;
			if (any(k) && j < n_train) {
				const ProposalCandidate* q =
				    pr.candidates + (size_t) (pr.phase + j * pr.stride) * pr.candidate_count + candidate(k);
				if (wide) {
					const uint2 v = load_pair_here(q);
					light[k] = (int) v.x;
					weight[k] = __uint_as_float(v.y);
				} else {
					light[k] = (int) load_here(&q->light);
					weight[k] = __uint_as_float(load_here(&q->pdf));
				}
			}
		}
	}
	RL_DEV void load_clusters(const MlpTrainParams& pr) {
#pragma unroll
		for (int k = 0; k != kBatch; ++k)
			cluster[k] = weight[k] > 0.0f && (uint32_t) light[k] < pr.light_count ? load_here(pr.light_cluster + light[k])
			                                                                     : kNoCluster;
	}
	// clusters: 0xffff for none.
	RL_DEV void stage(float* weights, uint16_t* clusters) const {
#pragma unroll
		for (int k = 0; k != kBatch; ++k)
			if (any(k)) {
				const int r = first + row(k), c = candidate(k);
				weights[staged_weight(c, r)] = weight[k];
				clusters[staged_cluster(c, r)] = (uint16_t) cluster[k];
			}
	}
};

// Adds `weights` of the `columns` FP32 columns of this thread's tensor-memory
// lane to the gradient at w (16-byte aligned, four per reduction) and the next
// column to *b; the rest is padding.  All threads call it; those without
// `active` add nothing.
RL_DEV void add_gradient(uint32_t taddr, int columns, float* w, int weights, float* b, bool active) {
	for (int col = 0; col != columns; col += 16) {
		uint32_t v[16];
		tc_load16(taddr + (uint32_t) col, v);
		tc_wait_load();
		if (!active) continue;
#pragma unroll
		for (int q = 0; q != 16; q += 4) {
			const float4 g = make_float4(__uint_as_float(v[q]), __uint_as_float(v[q + 1]), __uint_as_float(v[q + 2]),
			                             __uint_as_float(v[q + 3]));
			const int f = col + q;
			if (f + 4 <= weights) {
				if (g.x != 0.0f || g.y != 0.0f || g.z != 0.0f || g.w != 0.0f) atomicAdd(reinterpret_cast<float4*>(w + f), g);
				continue;
			}
			const float one[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
			for (int k = 0; k != 4; ++k)
				if (f + k <= weights && one[k] != 0.0f) atomicAdd(f + k < weights ? w + f + k : b, one[k]);
		}
	}
}

// The 16-byte words of an encoded row that part `part` of its threads writes
// start here: 5, 5, 4 and 4 of 18.
__host__ __device__ constexpr int part_first_word(int part) { return part <= 2 ? 5 * part : 2 + 4 * part; }
static_assert(part_first_word(kTtSplit) == kMlpFeatures / 8, "all words");

static __global__ void __launch_bounds__(kTtThreads, 1) mlp_train_tc_kernel(MlpTrainParams pr) {
	extern __shared__ __align__(1024) unsigned char tt_smem[];
	const int k_count = pr.k_count;
	const int k_pad = mlp_padded_clusters(k_count);
	const int chunks = (k_pad + kTcChunk - 1) / kTcChunk;
	const uint32_t dz_rows = (uint32_t) (k_pad / 8) * 128;  // DZ: bytes between 8-pixel groups
	const MlpLayout lay = mlp_layout(k_count);
	const uint32_t tid = threadIdx.x, warp = tid / 32;
	// Threads row, row + 128, ... share a row: part 0, 1, ... of its columns.
	const int row = (int) (tid % kTcRows), part = (int) (tid / kTcRows);
	const uint32_t base = smem_address(tt_smem);
	float* b1 = reinterpret_cast<float*>(tt_smem + kTtBias);
	float* b2 = b1 + kMlpHidden;
	float* b3 = b2 + kMlpHidden;
	for (int j = tid; j < kMlpHidden; j += kTtThreads) {
		b1[j] = pr.params[lay.b1 + j];
		b2[j] = pr.params[lay.b2 + j];
	}
	for (int j = tid; j < kTtMaxClusters; j += kTtThreads) b3[j] = j < k_count ? pr.params[lay.b3 + j] : 0.0f;
	// Columns 64..79 of H1 and H2: 1.0 then zeros (never overwritten).
	for (int idx = tid; idx < kTcRows * 16; idx += kTtThreads) {
		const int r = idx / 16, c = kMlpHidden + idx % 16;
		const __nv_bfloat16 v = __float2bfloat16_rn(c == kMlpHidden ? 1.0f : 0.0f);
		*reinterpret_cast<__nv_bfloat16*>(tt_smem + kTtH1 + tc_offset(r, c, kTtHiddenCols)) = v;
		*reinterpret_cast<__nv_bfloat16*>(tt_smem + kTtH2 + tc_offset(r, c, kTtHiddenCols)) = v;
	}
	const uint32_t bar = base + kTtBar, bar_weights = bar + 8;
	if (tid == 0) {
		for (int k = 0; k != 2; ++k) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar + 8 * k) : "memory");
		asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
		const uint32_t bytes = (uint32_t) mlp_weight_elements(k_count) * 2;
		mbarrier_expect_bytes(bar_weights, bytes);
		bulk_copy_to_shared(base + kTtW1, pr.weights, bytes, bar_weights);
	}
	if (warp == 0) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(base + kTtSlot),
		             "r"(kTtColumns)
		             : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
	}
	fence_async_shared();
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tt_smem + kTtSlot);
	const uint32_t lane_base = (warp % 4 * 32) << 16;
	float* const weights = reinterpret_cast<float*>(tt_smem + kTtD);
	uint16_t* const clusters = reinterpret_cast<uint16_t*>(tt_smem + kTtCluster);
	float* const part_sum = reinterpret_cast<float*>(tt_smem + kTtSum);                  // [part][row]
	__nv_bfloat16* const part_max = reinterpret_cast<__nv_bfloat16*>(tt_smem + kTtMax);  // [part][row]
	const uint32_t np = pr.width * pr.height;
	const uint32_t n_train = np > pr.phase ? (np - pr.phase + pr.stride - 1) / pr.stride : 0;
	const uint32_t tiles = (n_train + kTcRows - 1) / kTcRows;
	const int mc = pr.candidate_count;
	uint32_t parity = 0;
	bool product_pending = false;
	const bool weights_ok = __syncthreads_or(!tc_wait(bar_weights, 0)) == 0;
	bool failed = !weights_ok;
	auto issue = [&](auto products) {
		if (tid == 0 && !pr.skip_issue) {
			products();
			tc_commit(bar);
		}
	};
	// Products that the next issue's wait covers.
	auto issue_behind = [&](auto products) {
		if (tid == 0 && !pr.skip_issue) products();
	};
	auto await_products = [&] {
		const bool ok = tc_wait(bar, parity);
		parity ^= 1u;
		failed = __syncthreads_or(!ok) != 0;
		product_pending = failed && !pr.skip_issue;
		tc_fence_after();
	};
	auto sync_for_products = [&] {
		fence_async_shared();
		tc_fence_before();
		__syncthreads();
		tc_fence_after();
	};
	// This thread's part of the row's 64 transient columns + bias, ReLU, BF16
	// into H.
	constexpr int kHiddenPart = kMlpHidden / kTtSplit;
	static_assert(kHiddenPart == 16, "tc_load16");
	auto hidden_epilogue = [&](uint32_t h, const float* bias) {
		uint32_t v[kHiddenPart];
		tc_load16(tmem + lane_base + (uint32_t) (kHiddenPart * part), v);
		tc_wait_load();
		store_hidden(tt_smem + h, row, kHiddenPart * part, kTtHiddenCols, v, bias);
		sync_for_products();
	};
	// The same of the transient columns where H > 0, else 0, BF16 into the
	// DZ2/DZ1 buffer.
	auto gradient_epilogue = [&](uint32_t h) {
		const int c = kHiddenPart * part;
		uint32_t v[kHiddenPart];
		tc_load16(tmem + lane_base + (uint32_t) c, v);
		tc_wait_load();
#pragma unroll
		for (int q = 0; q != kHiddenPart / 8; ++q) {
			const uint4 act = *reinterpret_cast<const uint4*>(tt_smem + h + tc_offset(row, c + 8 * q, kTtHiddenCols));
			const uint32_t* a = &act.x;
			uint4 out;
			uint32_t* o = &out.x;
#pragma unroll
			for (int k = 0; k != 4; ++k) {
				const int j = 8 * q + 2 * k;
				o[k] = pack_bf16x2(bf16_lo(a[k]) > 0.0f ? __uint_as_float(v[j]) : 0.0f,
				                   bf16_hi(a[k]) > 0.0f ? __uint_as_float(v[j + 1]) : 0.0f);
			}
			*reinterpret_cast<uint4*>(tt_smem + kTtD + tc_offset(row, c + 8 * q, kMlpHidden)) = out;
		}
		sync_for_products();
	};
	// A tile's candidates and the inputs that this thread's words of a row need:
	// fetched while the backward products of the tile before run.
	constexpr int kWarpRows = kTcRows / (kTtThreads / 32);
	CandidateFetch<kWarpRows> fetch((int) warp * kWarpRows, mc);
	float x[kMlpInputs] = {};
	auto fetch_inputs = [&](uint32_t j0) {
		const uint32_t j = j0 + (uint32_t) row;
#pragma unroll
		for (int input = 0; input != kMlpInputs; ++input) {
			const int first = 8 * part_first_word(part), last = 8 * part_first_word(part + 1);  // features
			if (13 * input < last && 13 * input + 12 >= first)
				x[input] = __uint_as_float(
				    load_here(pr.gbuffer + (size_t) mlp_input_plane(input) * np + pr.phase + (size_t) min(j, n_train - 1) * pr.stride));
		}
	};
	if (blockIdx.x < tiles) {
		fetch.load_lights(pr, blockIdx.x * kTcRows, n_train);
		fetch.load_clusters(pr);
		fetch_inputs(blockIdx.x * kTcRows);
	}
	bool accumulated = false;  // the weight gradients in tensor memory hold at least one tile
	for (uint32_t tile = blockIdx.x; tile < tiles && !failed; tile += gridDim.x) {
		const uint32_t j0 = tile * kTcRows;
		// The row's training pixel: j0 + row.  Its inputs are encoded into E
		// (feature 130 is 1.0), a part of the row's words by each of its threads.
		const uint32_t my_j = j0 + (uint32_t) row, my_i = pr.phase + my_j * pr.stride;
		const bool in = my_j < n_train;
#pragma unroll
		for (int a = 0; a != 3; ++a) x[a] = (x[a] - pr.center[a]) * pr.inv_half_extent;
		if (part == 0) mlp_encode_row<part_first_word(0), part_first_word(1)>(tt_smem + kTtE, row, x, in, true);
		else if (part == 1) mlp_encode_row<part_first_word(1), part_first_word(2)>(tt_smem + kTtE, row, x, in, true);
		else if (part == 2) mlp_encode_row<part_first_word(2), part_first_word(3)>(tt_smem + kTtE, row, x, in, true);
		else mlp_encode_row<part_first_word(3), part_first_word(4)>(tt_smem + kTtE, row, x, in, true);
		fetch.stage(weights, clusters);
		sync_for_products();
		issue([&] {
			tc_mma_steps(tmem, tc_descriptor(base + kTtE, kMlpFeatures), 256, tc_descriptor(base + kTtW1, kMlpFeatures), 256,
			             tc_instruction(kTcRows, kMlpHidden), kMlpFeatures / 16, false);
		});
		const ProposalCandidate* cand = pr.candidates + (size_t) my_i * mc;
		const bool valid = in && !(pr.primitive && pr.primitive[my_i] == 0xffffffffu);
		int chosen = -1;
		float ss = 0.0f;
		if (valid && pr.shaded) {
			chosen = pr.records[my_i].x;
			ss = pr.shaded[my_i];
		}
		await_products();
		if (failed) break;
		hidden_epilogue(kTtH1, b1);
		issue([&] {
			tc_mma_steps(tmem, tc_descriptor(base + kTtH1, kTtHiddenCols), 256, tc_descriptor(base + kTtW2, kMlpHidden), 256,
			             tc_instruction(kTcRows, kMlpHidden), kMlpHidden / 16, false);
		});
		// While layer 2 runs, each thread goes over its row's candidates.
		float total = 0.0f;
		if (valid) {
#pragma unroll
			for (int c = 0; c != kTtHeld; c += 4) {
				const float4 w = *reinterpret_cast<const float4*>(weights + staged_weight(c, row));
				if (c < mc) total += w.x;
				if (c + 1 < mc) total += w.y;
				if (c + 2 < mc) total += w.z;
				if (c + 3 < mc) total += w.w;
			}
#pragma unroll 8
			for (int c = kTtHeld; c < mc; ++c) total += cand[c].pdf;
		}
		const bool learn = valid && total > 0.0f && total <= 3.0e38f;
		const float wu = pr.shaded ? 1.0f - pr.shadowed_weight : 1.0f;
		if (!learn) chosen = -1;
		ss = chosen >= 0 ? ss / (total / (float) mc) : 0.0f;
		if (pr.shaded) ss = pr.shadowed_weight * fminf(fmaxf(ss, 0.0f), 4.0f);
		const float coef = learn ? (wu + ss) * pr.inv_batch : 0.0f;
		const float unshadowed = wu / total * pr.inv_batch;
		// The candidates in this thread's columns.  (One candidate after another
		// for all parts, every warp would go through nearly all of them.)
		auto mine = [&](uint32_t cluster) { return (int) (cluster / 32 % kTtSplit) == part; };
		uint32_t todo = 0;
		if (learn) {
#pragma unroll
			for (int c = 0; c != kTtHeld; c += 8) {
				const uint4 packed = *reinterpret_cast<const uint4*>(clusters + staged_cluster(c, row));
				const uint32_t* w = &packed.x;
#pragma unroll
				for (int k = 0; k != 4; ++k) {
					const uint32_t lo = w[k] & 0xffffu, hi = w[k] >> 16;
					if (c + 2 * k < mc && lo != 0xffffu && mine(lo)) todo |= 1u << (c + 2 * k);
					if (c + 2 * k + 1 < mc && hi != 0xffffu && mine(hi)) todo |= 2u << (c + 2 * k);
				}
			}
		}
		await_products();
		if (failed) break;
		hidden_epilogue(kTtH2, b2);
		// Logits, 128 clusters per product, BF16; this thread's 32 of each
		// product stay in registers.  The row maximum.
		uint4 z[kTtMaxClusters / kTcChunk][4];
		float zmax = -INFINITY;
#pragma unroll
		for (int ch = 0; ch != kTtMaxClusters / kTcChunk; ++ch) {
			if (ch >= chunks) continue;
			const int c0 = ch * kTcChunk, n = min(kTcChunk, k_pad - c0);
			issue([&] {
				tc_mma_steps(tmem, tc_descriptor(base + kTtH2, kTtHiddenCols), 256,
				             tc_descriptor(base + kTtW3 + (uint32_t) c0 * 128, kMlpHidden), 256, tc_instruction(kTcRows, n),
				             kMlpHidden / 16, false);
			});
			await_products();
			if (failed) break;
			const int c = 32 * part;
#pragma unroll
			for (int g = 0; g != 2; ++g) {
				if (c + 16 * g >= n) continue;  // n is a multiple of 16
				uint32_t v[16];
				tc_load16(tmem + lane_base + (uint32_t) (c + 16 * g), v);
				tc_wait_load();
#pragma unroll
				for (int q = 0; q != 2; ++q) {
					const int col = c0 + c + 16 * g + 8 * q;
					if (col >= k_count) continue;  // k_count is a multiple of 8
					uint32_t* o = &z[ch][2 * g + q].x;
#pragma unroll
					for (int h = 0; h != 2; ++h) {
						const float4 b = *reinterpret_cast<const float4*>(b3 + col + 4 * h);
						const int j = 8 * q + 4 * h;
						o[2 * h] = pack_bf16x2(__uint_as_float(v[j]) + b.x, __uint_as_float(v[j + 1]) + b.y);
						o[2 * h + 1] = pack_bf16x2(__uint_as_float(v[j + 2]) + b.z, __uint_as_float(v[j + 3]) + b.w);
					}
#pragma unroll
					for (int k = 0; k != 4; ++k) zmax = fmaxf(zmax, fmaxf(bf16_lo(o[k]), bf16_hi(o[k])));
				}
			}
			part_max[kTcRows * part + row] = __float2bfloat16_rn(zmax);  // a BF16 value or -inf
			tc_fence_before();
			__syncthreads();
			tc_fence_after();
		}
		if (failed) break;
		// DZ = coef softmax(z), each thread on its columns of the row (zero for
		// padding clusters).
#pragma unroll
		for (int k = 0; k != kTtSplit; ++k) zmax = fmaxf(zmax, __bfloat162float(part_max[kTcRows * k + row]));
		float sum = 0.0f;
#pragma unroll
		for (int ch = 0; ch != kTtMaxClusters / kTcChunk; ++ch)
#pragma unroll
			for (int q = 0; q != 4; ++q)
				if (ch * kTcChunk + 32 * part + 8 * q < k_count) {
					const uint32_t* w = &z[ch][q].x;
#pragma unroll
					for (int k = 0; k != 4; ++k) sum += __expf(bf16_lo(w[k]) - zmax) + __expf(bf16_hi(w[k]) - zmax);
				}
		part_sum[kTcRows * part + row] = sum;
		__syncthreads();
		sum = part_sum[row];
#pragma unroll
		for (int k = 1; k != kTtSplit; ++k) sum += part_sum[kTcRows * k + row];
		const float scale = coef / sum;
#pragma unroll
		for (int ch = 0; ch != kTtMaxClusters / kTcChunk; ++ch)
#pragma unroll
			for (int q = 0; q != 4; ++q) {
				const int col = ch * kTcChunk + 32 * part + 8 * q;
				if (col >= k_pad) continue;
				uint4 out = make_uint4(0u, 0u, 0u, 0u);
				if (col < k_count) {
					const uint32_t* w = &z[ch][q].x;
					uint32_t* o = &out.x;
#pragma unroll
					for (int k = 0; k != 4; ++k)
						o[k] = pack_bf16x2(scale * __expf(bf16_lo(w[k]) - zmax), scale * __expf(bf16_hi(w[k]) - zmax));
				}
				*reinterpret_cast<uint4*>(tt_smem + kTtDz + tc_offset(row, col, k_pad)) = out;
			}
		const bool more = tile + gridDim.x < tiles;
		const uint32_t next_j0 = (tile + gridDim.x) * kTcRows;
		if (more) fetch.load_lights(pr, next_j0, n_train);
		// Minus the target, on this thread's columns: the candidates' weights
		// into their clusters, in order, the shadowed part into the chosen
		// light's.
		if (learn) {
			auto subtract = [&](uint32_t cluster, float target) {
				__nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(tt_smem + kTtDz + tc_offset(row, (int) cluster, k_pad));
				*d = __float2bfloat16_rn(__bfloat162float(*d) - target);
			};
			uint32_t cluster = 0;
			float w = 0.0f;
			auto next = [&] {  // the first one still to do
				const int c = todo ? __ffs(todo) - 1 : 0;
				cluster = clusters[staged_cluster(c, row)];
				w = weights[staged_weight(c, row)];
			};
			next();
			while (todo) {
				const uint32_t now = cluster;
				const float target = unshadowed * w;
				todo &= todo - 1;
				next();
				subtract(now, target);
			}
#pragma unroll 1
			for (int c = kTtHeld; c < mc; ++c) {
				const ProposalCandidate q = cand[c];
				const uint32_t cluster = candidate_cluster(pr, q.light, q.pdf);
				if (cluster != kNoCluster && mine(cluster)) subtract(cluster, unshadowed * q.pdf);
			}
			if (chosen >= 0 && (uint32_t) chosen < pr.light_count && ss > 0.0f) {
				const uint32_t cluster = pr.light_cluster[chosen];
				if (mine(cluster)) subtract(cluster, ss * pr.inv_batch);
			}
		}
		sync_for_products();
		// dh2 = DZ W3 (W3 read MN-major: N = hidden, K = clusters) and
		// dW3 += DZ^T [H2 | 1] (both MN-major, K = pixels).
		issue([&] {
			tc_mma_steps(tmem, tc_descriptor(base + kTtDz, k_pad), 256, tc_descriptor_mn(base + kTtW3, 1024, 128), 2048,
			             tc_instruction(kTcRows, kMlpHidden) | kTcBMajorMN, k_pad / 16, false);
		});
		issue_behind([&] {
			for (int ch = 0; ch != chunks; ++ch)
				tc_mma_steps(tmem + kTtGrad3 + 80 * ch, tc_descriptor_mn(base + kTtDz + 2048 * ch, dz_rows, 128), 2 * dz_rows,
				             tc_descriptor_mn(base + kTtH2, 1280, 128), 2 * 1280,
				             tc_instruction(kTcRows, kTtHiddenCols) | kTcAMajorMN | kTcBMajorMN, kTcRows / 16, accumulated);
		});
		// The candidates' clusters: a line per lane, thousands of cycles of L1
		// lookups, while the backward products run.
		if (more) fetch.load_clusters(pr);
		await_products();
		if (failed) break;
		gradient_epilogue(kTtH2);
		// dh1 = DZ2 W2 (W2 MN-major) and dW2 += DZ2^T [H1 | 1].
		issue([&] {
			tc_mma_steps(tmem, tc_descriptor(base + kTtD, kMlpHidden), 256, tc_descriptor_mn(base + kTtW2, 1024, 128), 2048,
			             tc_instruction(kTcRows, kMlpHidden) | kTcBMajorMN, kMlpHidden / 16, false);
			tc_mma_steps(tmem + kTtGrad2, tc_descriptor_mn(base + kTtD, 1024, 128), 2048,
			             tc_descriptor_mn(base + kTtH1, 1280, 128), 2 * 1280,
			             tc_instruction(kTcRows, kTtHiddenCols) | kTcAMajorMN | kTcBMajorMN, kTcRows / 16, accumulated);
		});
		if (more) fetch_inputs(next_j0);
		await_products();
		if (failed) break;
		gradient_epilogue(kTtH1);  // DZ1 replaces DZ2 (its products are done)
		// dW1 += DZ1^T E.
		issue([&] {
			tc_mma_steps(tmem + kTtGrad1, tc_descriptor_mn(base + kTtD, 1024, 128), 2048,
			             tc_descriptor_mn(base + kTtE, 2304, 128), 2 * 2304,
			             tc_instruction(kTcRows, kMlpFeatures) | kTcAMajorMN | kTcBMajorMN, kTcRows / 16, accumulated);
		});
		await_products();
		accumulated = true;
	}
	if (!failed && accumulated) {
		// Lane `row` of each accumulator: cluster (dW3) or hidden unit (dW2,
		// dW1); the parts take the accumulators in turn.
		for (int ch = part; ch < chunks; ch += kTtSplit) {
			const int c = ch * kTcChunk + row;
			add_gradient(tmem + lane_base + kTtGrad3 + 80 * ch, kTtHiddenCols, pr.grad + lay.w3 + (size_t) c * kMlpHidden,
			             kMlpHidden, pr.grad + lay.b3 + c, c < k_count);
		}
		if (part == 2)
			add_gradient(tmem + lane_base + kTtGrad2, kTtHiddenCols, pr.grad + lay.w2 + row * kMlpHidden, kMlpHidden,
			             pr.grad + lay.b2 + row, row < kMlpHidden);
		if (part == 3)
			add_gradient(tmem + lane_base + kTtGrad1, kMlpFeatures, pr.grad + lay.w1 + row * kMlpFeatures, kTtOnesFeature,
			             pr.grad + lay.b1 + row, row < kMlpHidden);
	}
	if (failed) {
		if (tid == 0) atomicOr(pr.error, kErrorTensorWait);
		if (product_pending) {
			tc_wait(bar, parity ^ 1u);
			if (tid == 0) tc_commit(bar);  // and products behind it
			tc_wait(bar, parity);
		}
		if (!weights_ok) tc_wait(bar_weights, 0);
	}
	tc_fence_before();
	__syncthreads();
	if (warp == 0) {
		tc_fence_after();
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kTtColumns) : "memory");
	}
}

}  // namespace risltc
