// mlp_train_tc_wide.cuh - online training of the proposal MLP on the tcgen05
// tensor cores for models of more than 256 clusters (up to 1024): the same
// training step as mlp_train_tc_kernel (forward pass, softmax cross-entropy
// gradient, backward products, weight gradients; BF16 operands, FP32
// accumulators), with the output layer taken in chunks of 128 clusters so
// that neither its weights nor its logits have to fit on chip at once.
//
// One CTA of 16 warps per SM takes tiles of 128 training pixels, four threads to
// a pixel, each with 32 columns of a chunk's rows.  W1 and W2 arrive in one bulk copy; W3 streams by chunk (16 KB each) into two shared
// buffers by bulk copies issued one chunk ahead.  Per tile:
//   D1 = E W1^T, H1 = ReLU(D1 + b1); D2 = H1 W2^T, H2 = ReLU(D2 + b2);
//   pass A, per chunk: its logits (BF16, as in inference) and the running
//     maximum and sum of exp(z - max) of each thread's columns (online
//     softmax), combined per row at the end;
//   pass B, per chunk: its logits again, DZ_c = coef exp(z - max) / sum in
//     BF16 minus the pixel's targets in this chunk (each subtraction rounded
//     to BF16, in candidate order, as in mlp_train_tc_kernel), then
//     dh2 += DZ_c W3_c (accumulated over the chunks in tensor memory) and
//     dW3_c = DZ_c^T [H2 | 1], added to the FP32 gradient with vector
//     atomics (the chunks' weight gradients do not fit in tensor memory);
//   DZ2 = dh2 * [H2 > 0]; dh1 = DZ2 W2 and dW2 += DZ2^T [H1 | 1];
//   DZ1 = dh1 * [H1 > 0]; dW1 += DZ1^T E (feature 130 of E is 1: db1).
// What bounds it: the chain of each chunk (product, two passes of exponentials,
// targets, products, 80 columns of atomics) at one tile per SM.  With a thread
// per pixel, four warps, a step of 259,200 pixels with 1,024 clusters and 32
// candidates took 4.17 ms, now 1.53; 129,600 pixels with 512 clusters 1.13 and
// 0.47 ms.  dW2 and dW1 accumulate in tensor memory over the CTA's tiles and are added
// once at the end.  Tensor memory (512 columns): 0..127 the per-tile
// products, 128..191 dh2, 192..271 dW3 of the current chunk, 272..351 dW2,
// 352..495 dW1.  Every wait is bounded (kTcWaitNs); on a timeout the kernel
// records kErrorTensorWait, waits (bounded) for its products and copies in
// flight, frees its tensor memory and returns.
#pragma once
#include "mlp_train_tc.cuh"

namespace risltc {

constexpr int kTwMaxClusters = 1024;
constexpr uint32_t kTwChunkBytes = kTcChunk * kMlpHidden * 2;  // one W3 chunk: 16 KB
constexpr uint32_t kTwDh2 = 128, kTwGrad3 = 192, kTwGrad2 = 272, kTwGrad1 = 352;
// Shared memory (bytes).
constexpr uint32_t kTwW1 = 0;
constexpr uint32_t kTwW2 = kTwW1 + kMlpHidden * kMlpFeatures * 2;
constexpr uint32_t kTwW3 = kTwW2 + kMlpHidden * kMlpHidden * 2;  // two chunk buffers
constexpr uint32_t kTwE = kTwW3 + 2 * kTwChunkBytes;
constexpr uint32_t kTwH1 = kTwE + kTcRows * kMlpFeatures * 2;
constexpr uint32_t kTwH2 = kTwH1 + kTcRows * kTtHiddenCols * 2;
constexpr uint32_t kTwDz = kTwH2 + kTcRows * kTtHiddenCols * 2;   // one chunk: 128 pixels x 128 clusters
constexpr uint32_t kTwD = kTwDz + kTcRows * kTcChunk * 2;         // DZ2, then DZ1
constexpr uint32_t kTwBias = kTwD + kTcRows * kMlpHidden * 2;     // b1, b2, b3 (FP32)
constexpr uint32_t kTwBar = kTwBias + (2 * kMlpHidden + kTwMaxClusters) * 4;  // products, W1W2, W3 buffers 0 and 1
constexpr uint32_t kTwSlot = kTwBar + 32;
// A tile's first kTtHeld candidates per row (weights, clusters) and the rows'
// sums and maxima by parts of the columns.
constexpr uint32_t kTwWeight = (kTwSlot + 8 + 15) / 16 * 16;
constexpr uint32_t kTwCluster = kTwWeight + kTtHeld * kTcRows * 4;
constexpr uint32_t kTwSum = kTwCluster + kTtHeld * kTcRows * 2;
constexpr uint32_t kTwMax = kTwSum + kTtSplit * kTcRows * 4;
constexpr uint32_t kTwSmemBytes = kTwMax + kTtSplit * kTcRows * 4;
// The M = 128 reads of DZ2 / DZ1 (MN-major, 64 real rows) reach past their
// buffer into the biases, as in mlp_train_tc_kernel.
static_assert(kTwBar - kTwD >= 14 * 1024 + 16 * 128 + 1024 + 128, "discarded rows stay in shared memory");
static_assert(kTwW3 % 1024 == 0 && kTwE % 1024 == 0 && kTwH1 % 1024 == 0 && kTwH2 % 1024 == 0 &&
                  kTwDz % 1024 == 0 && kTwD % 1024 == 0,
              "operand buffers 1 KB aligned");
static_assert(kTwSmemBytes <= 232448, "fits one CTA per SM");

static __global__ void __launch_bounds__(kTtThreads, 1) mlp_train_tc_wide_kernel(MlpTrainParams pr) {
	extern __shared__ __align__(1024) unsigned char tw_smem[];
	const int k_count = pr.k_count;
	const int k_pad = mlp_padded_clusters(k_count);
	const int chunks = (k_pad + kTcChunk - 1) / kTcChunk;
	const MlpLayout lay = mlp_layout(k_count);
	const uint32_t tid = threadIdx.x, warp = tid / 32;
	// Threads row, row + 128, ... share a row: part 0, 1, ... of its columns.
	const int row = (int) (tid % kTcRows), part = (int) (tid / kTcRows);
	float* const weights = reinterpret_cast<float*>(tw_smem + kTwWeight);
	uint16_t* const clusters = reinterpret_cast<uint16_t*>(tw_smem + kTwCluster);
	float* const part_sum = reinterpret_cast<float*>(tw_smem + kTwSum);  // [part][row]
	float* const part_max = reinterpret_cast<float*>(tw_smem + kTwMax);
	const uint32_t base = smem_address(tw_smem);
	float* b1 = reinterpret_cast<float*>(tw_smem + kTwBias);
	float* b2 = b1 + kMlpHidden;
	float* b3 = b2 + kMlpHidden;
	for (int j = tid; j < kMlpHidden; j += kTtThreads) {
		b1[j] = pr.params[lay.b1 + j];
		b2[j] = pr.params[lay.b2 + j];
	}
	for (int j = tid; j < kTwMaxClusters; j += kTtThreads) b3[j] = j < k_count ? pr.params[lay.b3 + j] : 0.0f;
	// Columns 64..79 of H1 and H2: 1.0 then zeros (never overwritten).
	for (int idx = tid; idx < kTcRows * 16; idx += kTtThreads) {
		const int r = idx / 16, c = kMlpHidden + idx % 16;
		const __nv_bfloat16 v = __float2bfloat16_rn(c == kMlpHidden ? 1.0f : 0.0f);
		*reinterpret_cast<__nv_bfloat16*>(tw_smem + kTwH1 + tc_offset(r, c, kTtHiddenCols)) = v;
		*reinterpret_cast<__nv_bfloat16*>(tw_smem + kTwH2 + tc_offset(r, c, kTtHiddenCols)) = v;
	}
	const uint32_t bar = base + kTwBar, bar_weights = bar + 8, bar_w3 = bar + 16;  // bar_w3 + 8 b: buffer b
	const char* w3_global = reinterpret_cast<const char*>(pr.weights) + kTwW3;  // W3 follows W1 and W2
	if (tid == 0) {
		for (int k = 0; k != 4; ++k) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar + 8 * k) : "memory");
		asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
		mbarrier_expect_bytes(bar_weights, kTwW3);
		bulk_copy_to_shared(base + kTwW1, pr.weights, kTwW3, bar_weights);
	}
	if (warp == 0) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(base + kTwSlot),
		             "r"(kTtColumns)
		             : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
	}
	fence_async_shared();
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tw_smem + kTwSlot);
	const uint32_t lane_base = (warp % 4 * 32) << 16;
	const uint32_t np = pr.width * pr.height;
	const uint32_t n_train = np > pr.phase ? (np - pr.phase + pr.stride - 1) / pr.stride : 0;
	const uint32_t tiles = (n_train + kTcRows - 1) / kTcRows;
	const int mc = pr.candidate_count;
	uint32_t parity = 0;
	bool product_pending = false;
	bool failed = __syncthreads_or(!tc_wait(bar_weights, 0)) != 0;
	const bool weights_ok = !failed;
	// W3 chunk copies: the seq-th copy of the CTA goes to buffer seq & 1 and
	// completes phase (seq >> 1) & 1 of that buffer's mbarrier.
	uint32_t copies_issued = 0, copies_waited = 0;
	auto copy_chunk = [&](int c) {
		if (tid == 0) {
			const uint32_t b = copies_issued & 1u;
			const uint32_t bytes = (uint32_t) min(kTcChunk, k_pad - c * kTcChunk) * kMlpHidden * 2;
			mbarrier_expect_bytes(bar_w3 + 8 * b, bytes);
			bulk_copy_to_shared(base + kTwW3 + b * kTwChunkBytes, w3_global + (size_t) c * kTwChunkBytes, bytes,
			                    bar_w3 + 8 * b);
		}
		++copies_issued;
	};
	// Waits for the oldest copy not yet waited for; returns its buffer's
	// shared address.
	auto await_chunk = [&]() -> uint32_t {
		const uint32_t b = copies_waited & 1u, ph = (copies_waited >> 1) & 1u;
		const bool ok = tc_wait(bar_w3 + 8 * b, ph);
		++copies_waited;
		failed = __syncthreads_or(!ok) != 0;
		return base + kTwW3 + b * kTwChunkBytes;
	};
	auto issue = [&](auto products) {
		if (tid == 0 && !pr.skip_issue) {
			products();
			tc_commit(bar);
		}
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
		store_hidden(tw_smem + h, row, kHiddenPart * part, kTtHiddenCols, v, bias);
		sync_for_products();
	};
	// The same of the 64 columns at `col` where H > 0, else 0, BF16 into D.
	auto gradient_epilogue = [&](uint32_t col, uint32_t h) {
		const int c = kHiddenPart * part;
		uint32_t v[kHiddenPart];
		tc_load16(tmem + lane_base + col + (uint32_t) c, v);
		tc_wait_load();
#pragma unroll
		for (int q = 0; q != kHiddenPart / 8; ++q) {
			const uint4 act = *reinterpret_cast<const uint4*>(tw_smem + h + tc_offset(row, c + 8 * q, kTtHiddenCols));
			const uint32_t* a = &act.x;
			uint4 out;
			uint32_t* o = &out.x;
#pragma unroll
			for (int k = 0; k != 4; ++k) {
				const int j = 8 * q + 2 * k;
				o[k] = pack_bf16x2(bf16_lo(a[k]) > 0.0f ? __uint_as_float(v[j]) : 0.0f,
				                   bf16_hi(a[k]) > 0.0f ? __uint_as_float(v[j + 1]) : 0.0f);
			}
			*reinterpret_cast<uint4*>(tw_smem + kTwD + tc_offset(row, c + 8 * q, kMlpHidden)) = out;
		}
		sync_for_products();
	};
	// Logits of chunk c (n clusters) into tensor-memory columns 0..n-1.
	auto logits_product = [&](uint32_t w3, int n) {
		issue([&] {
			tc_mma_steps(tmem, tc_descriptor(base + kTwH2, kTtHiddenCols), 256, tc_descriptor(w3, kMlpHidden), 256,
			             tc_instruction(kTcRows, n), kMlpHidden / 16, false);
		});
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
				x[input] = __uint_as_float(load_here(pr.gbuffer + (size_t) mlp_input_plane(input) * np + pr.phase +
				                                     (size_t) min(j, n_train - 1) * pr.stride));
		}
	};
	if (blockIdx.x < tiles) {
		fetch.load_lights(pr, blockIdx.x * kTcRows, n_train);
		fetch.load_clusters(pr);
		fetch_inputs(blockIdx.x * kTcRows);
	}
	bool accumulated = false;  // dW2 and dW1 in tensor memory hold at least one tile
	for (uint32_t tile = blockIdx.x; tile < tiles && !failed; tile += gridDim.x) {
		const uint32_t j0 = tile * kTcRows;
		const uint32_t my_j = j0 + (uint32_t) row, my_i = pr.phase + my_j * pr.stride;
		const bool in = my_j < n_train;
		copy_chunk(0);  // the tile's first W3 chunk, during layers 1 and 2
#pragma unroll
		for (int a = 0; a != 3; ++a) x[a] = (x[a] - pr.center[a]) * pr.inv_half_extent;
		if (part == 0) mlp_encode_row<part_first_word(0), part_first_word(1)>(tw_smem + kTwE, row, x, in, true);
		else if (part == 1) mlp_encode_row<part_first_word(1), part_first_word(2)>(tw_smem + kTwE, row, x, in, true);
		else if (part == 2) mlp_encode_row<part_first_word(2), part_first_word(3)>(tw_smem + kTwE, row, x, in, true);
		else mlp_encode_row<part_first_word(3), part_first_word(4)>(tw_smem + kTwE, row, x, in, true);
		fetch.stage(weights, clusters);
		sync_for_products();
		issue([&] {
			tc_mma_steps(tmem, tc_descriptor(base + kTwE, kMlpFeatures), 256, tc_descriptor(base + kTwW1, kMlpFeatures), 256,
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
		hidden_epilogue(kTwH1, b1);
		issue([&] {
			tc_mma_steps(tmem, tc_descriptor(base + kTwH1, kTtHiddenCols), 256, tc_descriptor(base + kTwW2, kMlpHidden), 256,
			             tc_instruction(kTcRows, kMlpHidden), kMlpHidden / 16, false);
		});
		// While layer 2 runs: the row's total candidate weight.
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
		await_products();
		if (failed) break;
		hidden_epilogue(kTwH2, b2);
		// Pass A: the maximum logit m and the sum of exp(z - m) of this thread's
		// columns of the row, 32 of each chunk.
		float zmax = -INFINITY, zsum = 0.0f, scale = 0.0f;
		const int cp = 32 * part;
		for (int u = 0; u != 2 * chunks && !failed; ++u) {
			const int ch = u % chunks, c0 = ch * kTcChunk, n = min(kTcChunk, k_pad - c0);
			const bool pass_b = u >= chunks;
			const uint32_t w3 = await_chunk();
			if (failed) break;
			if (u + 1 < 2 * chunks) copy_chunk((u + 1) % chunks);
			logits_product(w3, n);
			await_products();
			if (failed) break;
			// This thread's logits of the chunk, rounded to BF16.
			float z[32];
			if (cp < n) {
				uint32_t v[32];
				tc_load32(tmem + lane_base + (uint32_t) cp, v);
				tc_wait_load();
#pragma unroll
				for (int j = 0; j != 32; ++j)
					z[j] = cp + j < n && c0 + cp + j < k_count
					           ? __bfloat162float(__float2bfloat16_rn(__uint_as_float(v[j]) + b3[c0 + cp + j]))
					           : -INFINITY;
			}
			if (!pass_b) {
				if (cp < n) {
					float m = zmax;
#pragma unroll
					for (int j = 0; j != 32; ++j) m = fmaxf(m, z[j]);
					float s = zmax == -INFINITY ? 0.0f : zsum * __expf(zmax - m);
#pragma unroll
					for (int j = 0; j != 32; ++j)
						if (z[j] != -INFINITY) s += __expf(z[j] - m);
					zmax = m;
					zsum = s;
				}
				part_max[kTcRows * part + row] = zmax;
				part_sum[kTcRows * part + row] = zsum;
				tc_fence_before();
				__syncthreads();
				tc_fence_after();
				continue;
			}
			if (u == chunks) {  // the row's maximum and sum
#pragma unroll
				for (int k = 0; k != kTtSplit; ++k) zmax = fmaxf(zmax, part_max[kTcRows * k + row]);
				float sum = 0.0f;
#pragma unroll
				for (int k = 0; k != kTtSplit; ++k) {
					const float m = part_max[kTcRows * k + row];
					if (m != -INFINITY) sum += part_sum[kTcRows * k + row] * __expf(m - zmax);
				}
				scale = coef / sum;
			}
			// Pass B: DZ of this chunk, BF16, minus this chunk's targets, each
			// thread on its columns (zero for padding clusters).
#pragma unroll
			for (int q = 0; q != 4; ++q) {
				if (cp + 8 * q >= n) continue;
				uint4 out;
				uint32_t* o = &out.x;
#pragma unroll
				for (int k = 0; k != 4; ++k) {
					const int j = 8 * q + 2 * k;
					o[k] = pack_bf16x2(z[j] != -INFINITY ? scale * __expf(z[j] - zmax) : 0.0f,
					                   z[j + 1] != -INFINITY ? scale * __expf(z[j + 1] - zmax) : 0.0f);
				}
				*reinterpret_cast<uint4*>(tw_smem + kTwDz + tc_offset(row, cp + 8 * q, kTcChunk)) = out;
			}
			if (learn) {
				auto mine = [&](uint32_t cluster) { return cluster - (uint32_t) (c0 + cp) < (uint32_t) min(32, max(0, n - cp)); };
				auto subtract = [&](uint32_t cluster, float target) {
					__nv_bfloat16* zp =
					    reinterpret_cast<__nv_bfloat16*>(tw_smem + kTwDz + tc_offset(row, (int) cluster - c0, kTcChunk));
					*zp = __float2bfloat16_rn(__bfloat162float(*zp) - target);
				};
				uint32_t todo = 0;
#pragma unroll
				for (int c = 0; c != kTtHeld; c += 8) {
					const uint4 packed = *reinterpret_cast<const uint4*>(clusters + staged_cluster(c, row));
					const uint32_t* w = &packed.x;
#pragma unroll
					for (int k = 0; k != 4; ++k) {
						if (c + 2 * k < mc && mine(w[k] & 0xffffu)) todo |= 1u << (c + 2 * k);
						if (c + 2 * k + 1 < mc && mine(w[k] >> 16)) todo |= 2u << (c + 2 * k);
					}
				}
				for (; todo; todo &= todo - 1) {
					const int c = __ffs(todo) - 1;
					subtract(clusters[staged_cluster(c, row)], unshadowed * weights[staged_weight(c, row)]);
				}
#pragma unroll 1
				for (int c = kTtHeld; c < mc; ++c) {
					const ProposalCandidate q = cand[c];
					const uint32_t cluster = candidate_cluster(pr, q.light, q.pdf);
					if (mine(cluster)) subtract(cluster, unshadowed * q.pdf);
				}
				if (chosen >= 0 && (uint32_t) chosen < pr.light_count && ss > 0.0f) {
					const uint32_t cluster = pr.light_cluster[chosen];
					if (mine(cluster)) subtract(cluster, ss * pr.inv_batch);
				}
			}
			sync_for_products();
			// dh2 += DZ_c W3_c (W3 read MN-major: N = hidden, K = clusters)
			// and dW3_c = DZ_c^T [H2 | 1] (both MN-major, K = pixels).
			issue([&] {
				tc_mma_steps(tmem + kTwDh2, tc_descriptor(base + kTwDz, kTcChunk), 256, tc_descriptor_mn(w3, 1024, 128), 2048,
				             tc_instruction(kTcRows, kMlpHidden) | kTcBMajorMN, n / 16, ch > 0);
				tc_mma_steps(tmem + kTwGrad3, tc_descriptor_mn(base + kTwDz, 2048, 128), 2 * 2048,
				             tc_descriptor_mn(base + kTwH2, 1280, 128), 2 * 1280,
				             tc_instruction(kTcRows, kTtHiddenCols) | kTcAMajorMN | kTcBMajorMN, kTcRows / 16, false);
			});
			await_products();
			if (failed) break;
			// Lane `row` of dW3_c: cluster c0 + row; each part adds 16 weights to
			// the gradient (16-byte aligned rows of 64 floats), one the bias.
			const int cl = c0 + row;
			float* const w3_grad = pr.grad + lay.w3 + (size_t) cl * kMlpHidden;
			add_gradient(tmem + lane_base + kTwGrad3 + 16 * part, 16, w3_grad + 16 * part, 16, nullptr, cl < k_count);
			if (part == 0)
				add_gradient(tmem + lane_base + kTwGrad3 + kMlpHidden, 16, nullptr, 0, pr.grad + lay.b3 + cl, cl < k_count);
			tc_fence_before();
			__syncthreads();
			tc_fence_after();
		}
		if (failed) break;
		const bool more = tile + gridDim.x < tiles;
		const uint32_t next_j0 = (tile + gridDim.x) * kTcRows;
		if (more) fetch.load_lights(pr, next_j0, n_train);
		gradient_epilogue(kTwDh2, kTwH2);
		// dh1 = DZ2 W2 (W2 MN-major) and dW2 += DZ2^T [H1 | 1].
		issue([&] {
			tc_mma_steps(tmem, tc_descriptor(base + kTwD, kMlpHidden), 256, tc_descriptor_mn(base + kTwW2, 1024, 128), 2048,
			             tc_instruction(kTcRows, kMlpHidden) | kTcBMajorMN, kMlpHidden / 16, false);
			tc_mma_steps(tmem + kTwGrad2, tc_descriptor_mn(base + kTwD, 1024, 128), 2048,
			             tc_descriptor_mn(base + kTwH1, 1280, 128), 2 * 1280,
			             tc_instruction(kTcRows, kTtHiddenCols) | kTcAMajorMN | kTcBMajorMN, kTcRows / 16, accumulated);
		});
		if (more) fetch.load_clusters(pr);
		if (more) fetch_inputs(next_j0);
		await_products();
		if (failed) break;
		gradient_epilogue(0, kTwH1);  // DZ1 replaces DZ2 (its products are done)
		// dW1 += DZ1^T E.
		issue([&] {
			tc_mma_steps(tmem + kTwGrad1, tc_descriptor_mn(base + kTwD, 1024, 128), 2048,
			             tc_descriptor_mn(base + kTwE, 2304, 128), 2 * 2304,
			             tc_instruction(kTcRows, kMlpFeatures) | kTcAMajorMN | kTcBMajorMN, kTcRows / 16, accumulated);
		});
		await_products();
		accumulated = true;
	}
	if (!failed && accumulated) {
		if (part == 0)
			add_gradient(tmem + lane_base + kTwGrad2, kTtHiddenCols, pr.grad + lay.w2 + row * kMlpHidden, kMlpHidden,
			             pr.grad + lay.b2 + row, row < kMlpHidden);
		if (part == 1)
			add_gradient(tmem + lane_base + kTwGrad1, kMlpFeatures, pr.grad + lay.w1 + row * kMlpFeatures, kTtOnesFeature,
			             pr.grad + lay.b1 + row, row < kMlpHidden);
	}
	if (failed) {
		if (tid == 0) atomicOr(pr.error, kErrorTensorWait);
		if (product_pending) tc_wait(bar, parity ^ 1u);
		if (!weights_ok) tc_wait(bar_weights, 0);
	}
	// Every W3 copy issued completes before the CTA leaves (bounded waits).
	while (copies_waited != copies_issued) {
		const uint32_t b = copies_waited & 1u, ph = (copies_waited >> 1) & 1u;
		tc_wait(bar_w3 + 8 * b, ph);
		++copies_waited;
	}
	tc_fence_before();
	__syncthreads();
	if (warp == 0) {
		tc_fence_after();
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kTtColumns) : "memory");
	}
}

}  // namespace risltc
