// mlp_tc.cuh - the proposal MLP's forward pass on the 5th-generation tensor
// cores (tcgen05, sm_100 family).
//
// One CTA per SM holds the three weight matrices and works on up to four tiles
// of 128 pixels at once, one per group of four warps.  The encoded features
// (128 x 144), the hidden activations (128 x 64) and the weights live in
// shared memory as K-major BF16 operands in 8x8 core matrices (no swizzle);
// one thread of a group issues the products
//   D1 = A1 W1^T (K = 144), D2 = A2 W2^T (K = 64), D3 = A3 W3^T (K = 64,
//   up to 128 clusters per product)
// with FP32 accumulators in the group's 128 columns of tensor memory (each
// product replaces the one before, which the group has read by then), and each
// warp moves its 32 rows (pixels)
// from tensor memory to registers for the epilogues: bias, ReLU and BF16
// rounding back into shared memory for the next product, or bias and BF16
// rounding of the logits to global memory (as BF16 for the proposal kernel, or
// widened to FP32 for a caller of risltc_model_logits: a separate pass over
// 0.8 GB took 0.9 of that call's 1.1 ms at 960x540 with 256 clusters).  A
// tile is a chain of waits (inputs, four or more products, epilogues), so what
// counts is how many tiles an SM has in flight: that call takes 119 us with
// four sharing the weights, 127 us with two CTAs of one tile each.  Bounds now:
// its 531 MB of writes (78 us) and the shared-memory data pipe (half busy).
// Every wait on the tensor cores is bounded; on a timeout the kernel records
// kErrorTensorWait, waits once more (bounded) for its products in flight,
// frees its tensor memory and returns.
#pragma once
#include "mlp.cuh"

namespace risltc {

constexpr int kTcRows = 128;      // pixels per tile: M of every product
constexpr int kTcThreads = 128;   // warp w reads tensor-memory lanes 32w .. 32w + 31
constexpr int kTcChunk = 128;     // clusters per layer-3 product (N)
constexpr uint64_t kTcWaitNs = 1000000000ull;  // a tensor-core wait gives up after one second
constexpr uint32_t kErrorTensorWait = 1u << 2;  // error-word bit: a tensor-core wait ran out

RL_DEV uint32_t smem_address(const void* p) { return (uint32_t) __cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor of a K-major operand with k columns whose
// first core matrix is at shared address addr (no swizzle): core matrices
// 128 bytes apart along K (leading byte offset), 8-row groups (k / 8) * 128
// bytes apart (stride byte offset); bits 46-48 hold the descriptor version 1.
RL_DEV uint64_t tc_descriptor(uint32_t addr, int k) {
	const uint64_t leading = 128, stride = (uint64_t) (k >> 3) * 128;
	return (uint64_t) ((addr & 0x3FFFFu) >> 4) | ((leading >> 4) << 16) | ((stride >> 4) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, M x N.
__host__ __device__ constexpr uint32_t tc_instruction(int m, int n) {
	return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t) (n >> 3) << 17) | ((uint32_t) (m >> 4) << 24);
}

// D (tensor memory) = A B^T (+ D if accumulate).
RL_DEV void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t instruction, uint32_t accumulate) {
	asm volatile(
	    "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
	    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
	    :
	    : "r"(d), "l"(a), "l"(b), "r"(instruction), "r"(accumulate)
	    : "memory");
}

// `steps` products of consecutive 16-element steps along K: a and b are the
// first step's descriptors, a_step and b_step the bytes from one step to the
// next.  D starts from zero unless `accumulate`.  (Built anew for each product,
// the descriptors cost the issuing thread about 100 cycles a product.)
RL_DEV void tc_mma_steps(uint32_t d, uint64_t a, uint32_t a_step, uint64_t b, uint32_t b_step, uint32_t instruction,
                         int steps, bool accumulate) {
#pragma unroll 4
	for (int k = 0; k < steps; ++k) {
		tc_mma(d, a, b, instruction, accumulate || k > 0);
		a += a_step >> 4;
		b += b_step >> 4;
	}
}

// The mbarrier at shared address bar completes its phase when the products
// issued so far by this thread are done.
RL_DEV void tc_commit(uint32_t bar) {
	asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar)
	             : "memory");
}

RL_DEV bool mbarrier_try_wait(uint32_t bar, uint32_t parity) {
	uint32_t done;
	asm volatile(
	    "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
	    : "=r"(done)
	    : "r"(bar), "r"(parity)
	    : "memory");
	return done != 0;
}

RL_DEV uint64_t global_ns() {
	uint64_t t;
	asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
	return t;
}

// Waits for phase `parity` of the mbarrier for at most kTcWaitNs (and at
// most 2^28 polls).
RL_DEV bool tc_wait(uint32_t bar, uint32_t parity) {
	const uint64_t t0 = global_ns();
	for (uint32_t i = 0; i != (1u << 28); ++i) {
		if (mbarrier_try_wait(bar, parity)) return true;
		if ((i & 255u) == 255u && global_ns() - t0 > kTcWaitNs) return false;
	}
	return false;
}

// The mbarrier's phase also waits for `bytes` of asynchronous copies (one
// arrival by this thread).
RL_DEV void mbarrier_expect_bytes(uint32_t bar, uint32_t bytes) {
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}

// Bulk copy (TMA, no tensor map) of `bytes` (a multiple of 16; both
// addresses 16-byte aligned) from global memory into this CTA's shared
// memory, counted on the mbarrier.
RL_DEV void bulk_copy_to_shared(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
	             "l"(src), "r"(bytes), "r"(bar)
	             : "memory");
}

RL_DEV void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
RL_DEV void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
RL_DEV void tc_wait_load() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
// Makes this thread's shared-memory writes visible to the tensor cores.
RL_DEV void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// 32 consecutive FP32 columns of this thread's tensor-memory lane.
RL_DEV void tc_load32(uint32_t taddr, uint32_t (&v)[32]) {
	asm volatile(
	    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
	    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
	    : "r"(taddr));
}

// Row `row` of the encoded features (K-major, kMlpFeatures columns) from the
// pixel's ten inputs, eight BF16 columns per 16-byte store; zeros where the
// row holds no pixel.  Feature 130, the first padding one, is 1 with `ones`.
// (One two-byte store per feature took a sixth of the logits call: 191
// us at 960x540 with 256 clusters, 157 with these and the biases read
// four at a time.)
// kFirst, kLast: only the 16-byte words kFirst .. kLast - 1 of the row.
template <int kFirst = 0, int kLast = kMlpFeatures / 8>
RL_DEV void mlp_encode_row(unsigned char* rows, int row, const float (&x)[kMlpInputs], bool in, bool ones) {
	float low = 0.0f;
	uint32_t words[4] = {0u, 0u, 0u, 0u};
	auto put = [&](int f, float v) {  // f: compile-time constants, ascending
		if ((f & 1) == 0) {
			low = v;
			return;
		}
		words[(f >> 1) & 3] = pack_bf16x2(low, v);
		if ((f & 7) == 7 && f / 8 >= kFirst && f / 8 < kLast)
			*reinterpret_cast<uint4*>(rows + tc_offset(row, f - 7, kMlpFeatures)) =
			    make_uint4(words[0], words[1], words[2], words[3]);
	};
#pragma unroll
	for (int input = 0; input != kMlpInputs; ++input) {
		if (input * 13 + 12 < 8 * kFirst || input * 13 >= 8 * kLast) continue;
		float e[13];
		mlp_encode(x[input], e);
#pragma unroll
		for (int kind = 0; kind != 13; ++kind) put(input * 13 + kind, in ? e[kind] : 0.0f);
	}
#pragma unroll
	for (int f = kMlpInputs * 13; f != kMlpFeatures; ++f) put(f, ones && f == kMlpInputs * 13 ? 1.0f : 0.0f);
}

// kColumns columns from c on of row `row` of a hidden layer (K-major, k
// columns): the accumulators v plus the bias (16-byte aligned), ReLU, BF16.
template <int kColumns>
RL_DEV void store_hidden(unsigned char* hidden, int row, int c, int k, const uint32_t (&v)[kColumns], const float* bias) {
#pragma unroll
	for (int q = 0; q != kColumns / 8; ++q) {
		uint32_t o[4];
#pragma unroll
		for (int h = 0; h != 2; ++h) {
			const float4 b = *reinterpret_cast<const float4*>(bias + c + 8 * q + 4 * h);
			const int j = 8 * q + 4 * h;
			o[2 * h] = pack_bf16x2(fmaxf(__uint_as_float(v[j]) + b.x, 0.0f), fmaxf(__uint_as_float(v[j + 1]) + b.y, 0.0f));
			o[2 * h + 1] = pack_bf16x2(fmaxf(__uint_as_float(v[j + 2]) + b.z, 0.0f), fmaxf(__uint_as_float(v[j + 3]) + b.w, 0.0f));
		}
		*reinterpret_cast<uint4*>(hidden + tc_offset(row, c + 8 * q, k)) = make_uint4(o[0], o[1], o[2], o[3]);
	}
}

// Shared memory of the kernel for k_count clusters: W1, W2, W3 (rows padded
// to a multiple of 16; together the operand-layout weights of one bulk copy),
// the groups' buffers, the biases, two mbarriers per group (products, inputs),
// one for the weights and the tensor memory address.  A group's buffer holds
// its tile's encoded features (A1) and, once layer 1 has read them, the hidden
// activations (A2) at the same place and the staged logits behind those; after
// it the tile's 10 input rows (128 floats each), which arrive while the tile
// before is worked on.  As many groups as fit, up to kTcMaxGroups.
constexpr int kTcMaxGroups = 4;
constexpr uint32_t kTcA1Bytes = kTcRows * kMlpFeatures * 2, kTcA2Bytes = kTcRows * kMlpHidden * 2;
constexpr uint32_t kTcInputBytes = kMlpInputs * kTcRows * 4, kTcGroupBytes = kTcA1Bytes + kTcInputBytes;
constexpr uint32_t kTcSmemLimit = 232448;  // 227 KB
struct TcLayout {
	uint32_t w1, w2, w3, group, b1, b2, b3, bar, slot, total, weight_bytes, groups;
	int k_pad;
};
__host__ __device__ inline TcLayout tc_layout(int k_count) {
	TcLayout l;
	l.k_pad = mlp_padded_clusters(k_count);
	l.weight_bytes = (uint32_t) mlp_weight_elements(k_count) * 2;
	l.w1 = 0;
	l.w2 = l.w1 + kMlpHidden * kMlpFeatures * 2;
	l.w3 = l.w2 + kMlpHidden * kMlpHidden * 2;
	l.group = l.w3 + (uint32_t) l.k_pad * kMlpHidden * 2;
	const uint32_t rest = (2 * kMlpHidden + (uint32_t) l.k_pad) * 4 + (2 * kTcMaxGroups + 2) * 8;
	l.groups = (kTcSmemLimit - l.group - rest) / kTcGroupBytes;
	if (l.groups > kTcMaxGroups) l.groups = kTcMaxGroups;
	l.b1 = l.group + l.groups * kTcGroupBytes;
	l.b2 = l.b1 + kMlpHidden * 4;
	l.b3 = l.b2 + kMlpHidden * 4;
	l.bar = l.b3 + (uint32_t) l.k_pad * 4;
	l.slot = l.bar + (2 * kTcMaxGroups + 1) * 8;
	l.total = l.slot + 8;
	return l;
}

// G-buffer plane of MLP input k (position, normal, outgoing, roughness).
RL_DEV int mlp_input_plane(int k) { return k < 9 ? k : 16; }

// The logits' staging: rows of 128 bytes, 144 apart (lanes' 16-byte words of
// one index fall in distinct banks), from which a warp writes four rows per
// instruction.  (Each lane storing to its own row occupied the L1 data pipe
// for three quarters of the call: 157 us at 960x540 with 256 clusters, 127
// staged.  One bulk copy per row segment: 146 us with 256 bytes, 199 with 128,
// about 14 cycles per copy.)
constexpr int kLogitStage = 128, kLogitStride = 144;
static_assert(kTcA2Bytes + kTcRows * kLogitStride <= kTcA1Bytes, "a tile's staged logits fit behind its hidden activations");

// The barrier of a group's four warps, and the same with the OR of a predicate.
RL_DEV void group_sync(uint32_t group) { asm volatile("bar.sync %0, 128;\n" ::"r"(group + 1) : "memory"); }
RL_DEV bool group_any(uint32_t group, bool value) {
	uint32_t any;
	asm volatile(
	    "{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.or.pred q, %2, 128, p;\nselp.u32 %0, 1, 0, q;\n}\n"
	    : "=r"(any)
	    : "r"((uint32_t) value), "r"(group + 1)
	    : "memory");
	return any != 0;
}

template <bool kF32> struct LogitType {
	using type = __nv_bfloat16;
	RL_DEV static type* rows(const MlpParams& pr) { return pr.logits; }
};
template <> struct LogitType<true> {
	using type = float;
	RL_DEV static type* rows(const MlpParams& pr) { return pr.logits_f32; }
};

// kF32: the logits go to pr.logits_f32.
template <bool kF32> static __global__ void __launch_bounds__(kTcThreads * kTcMaxGroups, 1) mlp_logits_tc_kernel(MlpParams pr) {
	extern __shared__ __align__(1024) unsigned char tc_smem[];
	const int k_count = pr.k_count;
	const MlpLayout lay = mlp_layout(k_count);
	const TcLayout tl = tc_layout(k_count);
	// Group g (four warps) has its own tiles; thread tid of it takes row tid.
	const uint32_t group = threadIdx.x / kTcThreads, tid = threadIdx.x % kTcThreads, warp = tid / 32;
	const uint32_t base = smem_address(tc_smem);
	float* b1 = reinterpret_cast<float*>(tc_smem + tl.b1);
	float* b2 = reinterpret_cast<float*>(tc_smem + tl.b2);
	float* b3 = reinterpret_cast<float*>(tc_smem + tl.b3);
	const uint32_t a1 = tl.group + group * kTcGroupBytes, a2 = a1, stage = a2 + kTcA2Bytes, in = a1 + kTcA1Bytes;
	const float* inputs = reinterpret_cast<const float*>(tc_smem + in);  // [10][128]
	for (uint32_t j = threadIdx.x; j < (uint32_t) kMlpHidden; j += blockDim.x) {
		b1[j] = pr.params[lay.b1 + j];
		b2[j] = pr.params[lay.b2 + j];
	}
	for (int j = (int) threadIdx.x; j < tl.k_pad; j += (int) blockDim.x) b3[j] = j < k_count ? pr.params[lay.b3 + j] : 0.0f;
	const uint32_t bar_weights = base + tl.bar, bar = bar_weights + 8 + 16 * group, bar_inputs = bar + 8;
	const uint32_t np = pr.width * pr.height;
	const uint32_t tiles = (np + kTcRows - 1) / kTcRows;
	// A tile's input rows come by bulk copy when every row is 16-byte aligned
	// and a multiple of 16 bytes long, else by plain loads.
	const bool bulk_inputs = np % 4 == 0 && (reinterpret_cast<uintptr_t>(pr.gbuffer) & 15) == 0;
	// Bulk copies issued and waited for on the inputs' mbarrier (the same on
	// every thread: the issue decisions are uniform).
	uint32_t inputs_issued = 0, inputs_waited = 0;
	auto fetch_inputs = [&](uint32_t tile) {
		if (tid == 0) {
			const uint32_t p0 = tile * kTcRows, rows = min((uint32_t) kTcRows, np - p0);
			mbarrier_expect_bytes(bar_inputs, kMlpInputs * rows * 4);
			for (int k = 0; k != kMlpInputs; ++k)
				bulk_copy_to_shared(base + in + k * kTcRows * 4, pr.gbuffer + (size_t) mlp_input_plane(k) * np + p0,
				                    rows * 4, bar_inputs);
		}
		++inputs_issued;
	};
	if (threadIdx.x == 0) {
		for (uint32_t i = 0; i != 1 + 2 * tl.groups; ++i)
			asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar_weights + 8 * i) : "memory");
		asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
		// The weights in one bulk copy.
		mbarrier_expect_bytes(bar_weights, tl.weight_bytes);
		bulk_copy_to_shared(base + tl.w1, pr.weights, tl.weight_bytes, bar_weights);
	}
	const uint32_t columns = tl.groups > 2 ? 512u : tl.groups * 128u;  // a power of two
	if (threadIdx.x < 32) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(base + tl.slot),
		             "r"(columns)
		             : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
	}
	fence_async_shared();
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tc_smem + tl.slot);
	const uint32_t d = tmem + 128 * group;  // the group's products, one after another
	const uint32_t first_tile = blockIdx.x + group * gridDim.x, tile_step = gridDim.x * tl.groups;
	if (bulk_inputs && first_tile < tiles) fetch_inputs(first_tile);  // the first tile's inputs
	const uint32_t lane_base = (warp * 32) << 16;  // this warp's tensor-memory lanes
	uint32_t parity = 0;
	bool product_pending = false;
	const bool weights_ok = __syncthreads_or(!tc_wait(bar_weights, 0)) == 0;
	bool failed = !weights_ok;
	// Products in a row: issued by the group's thread 0, then all of its threads
	// wait for them.  With pr.skip_issue (fault injection) nothing is issued or committed, so
	// the wait runs out.
	auto run = [&](auto issue) {
		if (tid == 0 && !pr.skip_issue) {
			issue();
			tc_commit(bar);
		}
		const bool ok = tc_wait(bar, parity);
		parity ^= 1u;
		failed = group_any(group, !ok);
		product_pending = failed && !pr.skip_issue;
		tc_fence_after();
	};
	// Epilogue of a hidden layer: row tid of D (64 columns) + bias, ReLU,
	// BF16 into A2.
	auto hidden_epilogue = [&](const float* bias) {
		for (int c = 0; c != kMlpHidden; c += 32) {
			uint32_t v[32];
			tc_load32(d + lane_base + (uint32_t) c, v);
			tc_wait_load();
			store_hidden(tc_smem + a2, (int) tid, c, kMlpHidden, v, bias);
		}
		fence_async_shared();
		tc_fence_before();
		group_sync(group);
		tc_fence_after();
	};
	using Out = typename LogitType<kF32>::type;
	Out* const logits = LogitType<kF32>::rows(pr);
	constexpr int kStage = kLogitStage / (int) sizeof(Out);  // columns
	constexpr uint32_t kWords = kLogitStage / 16;
	const bool wide_stores = (reinterpret_cast<uintptr_t>(logits) & 15) == 0;
	for (uint32_t tile = first_tile; tile < tiles && !failed; tile += tile_step) {
		const uint32_t p0 = tile * kTcRows;
		if (bulk_inputs) {
			// This tile's input rows (issued during the previous tile).
			failed = group_any(group, !tc_wait(bar_inputs, inputs_waited & 1u));
			if (failed) break;
			++inputs_waited;
		}
		// Encode the tile's pixels into A1: thread tid takes row tid.
		{
			const uint32_t i = p0 + tid;
			float x[kMlpInputs];
#pragma unroll
			for (int input = 0; input != kMlpInputs; ++input) {
				x[input] = 0.0f;
				if (i < np && bulk_inputs) {
					x[input] = inputs[input * kTcRows + tid];
					if (input < 3) x[input] = (x[input] - pr.center[input]) * pr.inv_half_extent;
				} else if (i < np) {
					x[input] = mlp_input(pr.gbuffer, np, i, pr.center, pr.inv_half_extent, input);
				}
			}
			mlp_encode_row(tc_smem + a1, (int) tid, x, i < np, false);
		}
		fence_async_shared();
		tc_fence_before();
		group_sync(group);
		tc_fence_after();
		// The inputs are encoded: the next tile's arrive while this one is worked on.
		if (bulk_inputs && tile + tile_step < tiles) fetch_inputs(tile + tile_step);
		run([&] {
			tc_mma_steps(d, tc_descriptor(base + a1, kMlpFeatures), 256, tc_descriptor(base + tl.w1, kMlpFeatures), 256,
			             tc_instruction(kTcRows, kMlpHidden), kMlpFeatures / 16, false);
		});
		if (failed) break;
		hidden_epilogue(b1);
		run([&] {
			tc_mma_steps(d, tc_descriptor(base + a2, kMlpHidden), 256, tc_descriptor(base + tl.w2, kMlpHidden), 256,
			             tc_instruction(kTcRows, kMlpHidden), kMlpHidden / 16, false);
		});
		if (failed) break;
		hidden_epilogue(b2);
		for (int c0 = 0; c0 < tl.k_pad && !failed; c0 += kTcChunk) {
			const int n = min(kTcChunk, tl.k_pad - c0);
			run([&] {
				tc_mma_steps(d, tc_descriptor(base + a2, kMlpHidden), 256,
				             tc_descriptor(base + tl.w3 + (uint32_t) c0 * 128, kMlpHidden), 256, tc_instruction(kTcRows, n),
				             kMlpHidden / 16, false);
			});
			if (failed) break;
			for (int c = 0; c < n; c += 32) {
				uint32_t v[32];
				tc_load32(d + lane_base + (uint32_t) c, v);
				tc_wait_load();
				const int at = c % kStage;  // of the staged columns
				unsigned char* const staged = tc_smem + stage + tid * kLogitStride + at * (int) sizeof(Out);
#pragma unroll
				for (int q = 0; q != 4; ++q) {
					const int j0 = c0 + c + 8 * q;
					if (j0 + 8 > k_count) continue;  // k_count is a multiple of 8
					uint32_t o[4];
#pragma unroll
					for (int h = 0; h != 2; ++h) {
						const float4 b = *reinterpret_cast<const float4*>(b3 + j0 + 4 * h);
						const int j = 8 * q + 4 * h;
						o[2 * h] = pack_bf16x2(__uint_as_float(v[j]) + b.x, __uint_as_float(v[j + 1]) + b.y);
						o[2 * h + 1] = pack_bf16x2(__uint_as_float(v[j + 2]) + b.z, __uint_as_float(v[j + 3]) + b.w);
					}
					if (!kF32) {
						*reinterpret_cast<uint4*>(staged + 16 * q) = make_uint4(o[0], o[1], o[2], o[3]);
					} else {
#pragma unroll
						for (int h = 0; h != 2; ++h)
							*reinterpret_cast<uint4*>(staged + 32 * q + 16 * h) =
							    make_uint4(o[2 * h] << 16, o[2 * h] & 0xffff0000u, o[2 * h + 1] << 16, o[2 * h + 1] & 0xffff0000u);
					}
				}
				// With the stage full (or its last columns in it) the warp
				// writes its rows' columns first .. end - 1, four rows of up to
				// 128 bytes at a time.
				const int first = c0 + c - at, end = min(c0 + c + 32, k_count);
				if ((at + 32 != kStage && c + 32 < n) || end <= first) continue;
				__syncwarp();
				const unsigned char* const rows = tc_smem + stage + (tid & ~31u) * kLogitStride;
				const uint32_t row0 = p0 + (tid & ~31u);
				if (wide_stores) {
					const int word = (int) (tid % kWords);
					const bool mine = 16 * word < (end - first) * (int) sizeof(Out);
#pragma unroll 4
					for (uint32_t r = tid % 32 / kWords; r < 32; r += 32 / kWords)
						if (mine && row0 + r < np)
							*reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(logits + (size_t) (row0 + r) * k_count + first) + 16 * word) =
							    *reinterpret_cast<const uint4*>(rows + r * kLogitStride + 16 * word);
				} else {
					for (uint32_t r = 0; r != 32 && row0 + r < np; ++r)
						for (int k = (int) (tid % 32); k < end - first; k += 32)
							logits[(size_t) (row0 + r) * k_count + first + k] =
							    reinterpret_cast<const Out*>(rows + r * kLogitStride)[k];
				}
				__syncwarp();
			}
			tc_fence_before();
			group_sync(group);
			tc_fence_after();
		}
	}
	if (failed) {
		// Record the timeout, then wait (bounded) for whatever is still in
		// flight: a product, the weights' copy, input copies.
		if (tid == 0) atomicOr(pr.error, kErrorTensorWait);
		if (product_pending) tc_wait(bar, parity ^ 1u);
		if (!weights_ok) tc_wait(bar_weights, 0);
		while (inputs_waited < inputs_issued) tc_wait(bar_inputs, inputs_waited++ & 1u);
	}
	tc_fence_before();
	__syncthreads();
	if (threadIdx.x < 32) {
		tc_fence_after();
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(columns) : "memory");
	}
}

}  // namespace risltc
