// Router for larger batches on tcgen05: logits = x . W_r^T (mlx/src/nn/moe.rs:67), softmax and top-k (:70-82), the
// shared expert's gate (:174-177) and the fp16 copy of x, for a tile of 32, 64 or 128 tokens and all experts per CTA.
//
// The router's rows are the A operand (M = 128 experts, one or two accumulators), the tile's tokens the N side, K in
// steps of 64, both operands by tiled TMA through a ring of four to six stages.  What bounds it is bringing all of W_r
// (1 MB at 256 experts of 2048) into every SM, so that the tile is the smallest that covers the batch in one wave: a
// larger one reads W_r less often, a smaller one leaves fewer SMs idle and finishes its tokens' top-k sooner.
// The mma.sync kernel this replaces moved the same tiles by cp.async in two buffers for 32 tokens a CTA, and copied
// x after the product instead of beside it.  256 experts of 2048 on a B200: 8192 tokens 79 -> 51 us, 1777 tokens
// 57 -> 45, 16384 tokens 147 -> 96.
//
// Sixteen warps: 0 issues the MMAs, 1 owns tensor memory, 2 loads, 4..7 move the logits (lane = expert, column =
// token) into shared memory, 8..15 write the fp16 copy and the gate while the product runs; then all take tokens'
// softmax and top-k.  Every wait is bounded.  On expiry the CTA waits for its copies and MMAs in flight, frees tensor
// memory, sets the caller's status word where there is one, and gives its tokens experts 0 .. k-1 (valid, whatever is done
// with them next) with NaN weights, which no result can hide.
#include <atomic>

#include "route_common.cuh"
#include "tcgen05.cuh"

namespace imx {

namespace {

using namespace route;
using namespace tc;

constexpr int kRtThreads = 512;
constexpr int kRtK = 64;
constexpr int kRtMaxStages = 6;
constexpr int kRtMaxExperts = 256;
constexpr size_t kRtSmemMost = 227 * 1024;
std::atomic<int> g_route_spin_limit{kSpin};

struct RtBars {
    uint64_t full[kRtMaxStages];
    uint64_t empty[kRtMaxStages];
    uint64_t acc_full;
    uint64_t retired;                              // after an expired wait: the MMAs issued before it
    uint32_t tmem_base;
    int abort;
};

struct RtMaps {
    CUtensorMap x, w;
};

template <int NTOK>
__global__ void __launch_bounds__(kRtThreads, 1)
route_tc_kernel(const __nv_bfloat16* __restrict__ x, int n_tokens, int H, int E, const float* __restrict__ logit_bias, int k,
                int norm, const __nv_bfloat16* __restrict__ w_sg, int32_t* __restrict__ topk_idx, float* __restrict__ topk_w,
                float* __restrict__ shared_gate, __half* __restrict__ x16, const int obits, const float pair_scale_odd,
                const int stages, const int spin_limit, int32_t* __restrict__ status, const __grid_constant__ RtMaps maps) {
    constexpr uint32_t kTmem = 2 * NTOK;                     // columns: two accumulators of NTOK
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int halves = E > 128 ? 2 : 1;
    const uint32_t w_bytes = (uint32_t)halves * 128u * kRtK * 2u;
    const uint32_t stage_bytes = w_bytes + NTOK * kRtK * 2;
    RtBars* bars = reinterpret_cast<RtBars*>(base + (size_t)stages * stage_bytes);
    float* s_logits = reinterpret_cast<float*>(base);        // [NTOK][E], in the stages' place once the product is done
    const uint32_t sbase = smem_u32(base);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tok0 = blockIdx.x * NTOK;
    const int ksteps = H / kRtK;
    volatile int* abort_flag = &bars->abort;

    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(smem_u32(&bars->full[s]), 1);
            mbar_init(smem_u32(&bars->empty[s]), 1);
        }
        mbar_init(smem_u32(&bars->acc_full), 1);
        mbar_init(smem_u32(&bars->retired), 1);
        bars->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)),
                     "r"(kTmem)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    int copied = 0;                                          // K steps the loader has started

    if (warp == 0) {
        int s = 0;
        uint32_t ph = 0;
        // bf16 x bf16 -> fp32
        const uint32_t idesc = idesc_for(128, NTOK) | (1u << 7) | (1u << 10);
        for (int ks = 0; ks < ksteps; ++ks) {
            if (!mbar_wait(smem_u32(&bars->full[s]), ph, abort_flag, spin_limit)) break;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t stage = sbase + (uint32_t)s * stage_bytes;
                for (int h = 0; h < halves; ++h)
#pragma unroll
                    for (int kk = 0; kk < kRtK / 16; ++kk)
                        umma_ss(tmem + (uint32_t)(h * NTOK), smem_desc(stage + (uint32_t)h * 16384u) + 2 * kk,
                                smem_desc(stage + w_bytes) + 2 * kk, idesc, (ks > 0 || kk > 0) ? 1u : 0u);
                umma_commit(smem_u32(&bars->empty[s]));
                if (ks == ksteps - 1) umma_commit(smem_u32(&bars->acc_full));
            }
            __syncwarp();
            if (++s == stages) {
                s = 0;
                ph ^= 1u;
            }
        }
    } else if (warp == 2) {
        int s = 0;
        uint32_t ph = 0;
        for (int ks = 0; ks < ksteps; ++ks, ++copied) {
            if (!mbar_wait(smem_u32(&bars->empty[s]), ph ^ 1u, abort_flag, spin_limit)) break;
            if (lane == 0) {
                const uint32_t stage = sbase + (uint32_t)s * stage_bytes, bar = smem_u32(&bars->full[s]);
                mbar_expect_tx(bar, stage_bytes);
                for (int h = 0; h < halves; ++h) tma_load_2d(stage + (uint32_t)h * 16384u, &maps.w, ks * kRtK, h * 128, bar);
                tma_load_2d(stage + w_bytes, &maps.x, ks * kRtK, tok0, bar);
            }
            __syncwarp();
            if (++s == stages) {
                s = 0;
                ph ^= 1u;
            }
        }
    } else if (warp >= 4 && warp < 8) {
        if (mbar_wait(smem_u32(&bars->acc_full), 0u, abort_flag, spin_limit)) {
            tc_fence_after();
            const int q = warp & 3;
            for (int h = 0; h < halves; ++h) {
                const int e = h * 128 + q * 32 + lane;
                const float b = logit_bias != nullptr && e < E ? logit_bias[e] : 0.f;
                for (int c = 0; c < NTOK / 32; ++c) {
                    uint32_t v[32];
                    tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(h * NTOK + c * 32), v);
                    if (e < E) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) s_logits[(size_t)(c * 32 + i) * E + e] = __uint_as_float(v[i]) + b;
                    }
                }
            }
            tc_fence_before();
        }
    } else if (warp >= 8) {
        for (int r = warp - 8; r < NTOK; r += 8) {
            const int tok = tok0 + r;
            if (tok >= n_tokens) break;
            const __nv_bfloat16* xr = x + (size_t)tok * H;
            if (x16 != nullptr) {
                // a block of 16 per lane at a time, in the order the expert kernels of this code width read
                __half* dst = x16 + (size_t)tok * H;
#pragma unroll 4
                for (int c = lane * 16; c < H; c += 32 * 16) convert_block16(obits, xr + c, dst + c, pair_scale_odd);
            }
            if (w_sg != nullptr) {
                float acc_g = 0.f;
                for (int c = lane * 8; c < H; c += 256) {
                    const uint4 xv = __ldg(reinterpret_cast<const uint4*>(xr + c));
                    const uint4 wv = __ldg(reinterpret_cast<const uint4*>(w_sg + c));
                    const __nv_bfloat162* xb = reinterpret_cast<const __nv_bfloat162*>(&xv);
                    const __nv_bfloat162* wb = reinterpret_cast<const __nv_bfloat162*>(&wv);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 xf = __bfloat1622float2(xb[i]), wf = __bfloat1622float2(wb[i]);
                        acc_g = fmaf(xf.x, wf.x, acc_g);
                        acc_g = fmaf(xf.y, wf.y, acc_g);
                    }
                }
                acc_g = warp_sum(acc_g);
                if (lane == 0) shared_gate[tok] = 1.0f / (1.0f + expf(-acc_g));
            }
        }
    }
    __syncthreads();
    const bool gave_up = bars->abort != 0;
    if (gave_up) {
        if (warp == 0) {
            if (elect_one()) umma_commit(smem_u32(&bars->retired));
            __syncwarp();
            mbar_drain(smem_u32(&bars->retired), 0u);
        } else if (warp == 2) {
            for (int ks = max(0, copied - stages); ks < copied; ++ks)
                mbar_drain(smem_u32(&bars->full[ks % stages]), (uint32_t)(ks / stages) & 1u);
        }
        __syncthreads();
    }
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmem) : "memory");
    if (gave_up) {
        if (tid == 0 && status != nullptr) atomicExch(status, 3);
        const long first = (long)tok0 * k, last = (long)min(n_tokens, tok0 + NTOK) * k;
        for (long i = first + tid; i < last; i += kRtThreads) {
            topk_idx[i] = (int32_t)((i - first) % k);
            topk_w[i] = __uint_as_float(0x7fc00000u);
        }
        return;
    }
    for (int r = warp; r < NTOK; r += kRtThreads / 32) {
        const int tok = tok0 + r;
        if (tok >= n_tokens) break;
        const float* lg = s_logits + (size_t)r * E;
        int32_t* oi = topk_idx + (size_t)tok * k;
        float* ow = topk_w + (size_t)tok * k;
        if (E <= 32) softmax_topk_warp<1>(lg, E, k, norm, oi, ow);
        else if (E <= 64) softmax_topk_warp<2>(lg, E, k, norm, oi, ow);
        else if (E <= 128) softmax_topk_warp<4>(lg, E, k, norm, oi, ow);
        else softmax_topk_warp<8>(lg, E, k, norm, oi, ow);
    }
}

template <int NTOK>
int launch_tile(const void* x, int n, int H, const void* Wr, const float* logit_bias, int E, int k, int norm, const void* w_sg,
                int32_t* topk_idx, float* topk_w, float* shared_gate, void* x16, const Order16& order, int32_t* status,
                cudaStream_t stream) {
    const size_t stage = (size_t)(E > 128 ? 2 : 1) * 128 * kRtK * 2 + (size_t)NTOK * kRtK * 2;
    const size_t fixed = sizeof(RtBars) + 1024;
    int stages = (int)((kRtSmemMost - fixed) / stage);
    if (stages > kRtMaxStages) stages = kRtMaxStages;
    size_t ring = (size_t)stages * stage;
    IMX_REQUIRE((size_t)NTOK * E * sizeof(float) <= ring, "route: the logits of a tile exceed the ring");
    RtMaps maps;
    IMX_TRY(make_tensor_map_2d(x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (size_t)n, (size_t)H, (size_t)H * 2, kRtK, NTOK, true, &maps.x));
    IMX_TRY(make_tensor_map_2d(Wr, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (size_t)E, (size_t)H, (size_t)H * 2, kRtK, 128, true, &maps.w));
    route_tc_kernel<NTOK><<<ceil_div(n, NTOK), kRtThreads, ring + fixed, stream>>>(
        (const __nv_bfloat16*)x, n, H, E, logit_bias, k, norm, (const __nv_bfloat16*)w_sg, topk_idx, topk_w, shared_gate,
        (__half*)x16, order_bits(order), order.pair_scale_odd, stages, g_route_spin_limit.load(), status, maps); IMX_LAUNCHED();
    IMX_CHECK_CUDA(cudaGetLastError());
    return IMX_OK;
}

}  // namespace

// Test hook (include/ironmlx_b200_testing.h).
void testing_route_give_up(int on) { g_route_spin_limit.store(on ? 0 : kSpin); }

// A tile takes all K steps one after the other whatever the batch (15 us at a hidden size of 512, 29 at 2048, 73 at 9728),
// the cluster-per-token kernel's time grows with the tokens and, less, with the experts; it serves the batches that this
// one would spread over a few CTAs.  Both on a B200, cluster / this one, us: 16 experts of 512, 256 tokens 9.2 / 15.2, 400
// 13.3 / 14.6, 700 17.4 / 15.4; 16 of 2048, 700 tokens 22.7 / 28.6, 1024 28.5 / 28.7, 1400 33.8 / 28.8; 60 of 1024, 256 tokens
// 14.5 / 18.3, 400 20.4 / 18.3; 60 of 2048, 400 tokens 26.4 / 30.8, 700 34.9 / 30.9.
static bool enough_tokens(int n, int H, int E) { return (long)n * (E + 40) >= (H <= 1024 ? 30000L : 52000L); }

bool route_tc_supported(const void* x, int n, int H, const void* Wr, int E, const void* x16, const Order16& order) {
    return n >= 256 && enough_tokens(n, H, E) && H % kRtK == 0 && E <= kRtMaxExperts && (((uintptr_t)x | (uintptr_t)Wr | (uintptr_t)x16) % 16) == 0 &&
           order_bits(order) >= 0;
}

int launch_route_tc(const void* x, int n, int H, const void* Wr, const float* logit_bias, int E, int k, int norm, const void* w_sg,
                    int32_t* topk_idx, float* topk_w, float* shared_gate, void* x16, const Order16& order, int32_t* status,
                    cudaStream_t stream) {
    DeviceInfo di;
    IMX_TRY(current_device(&di));
    if (device_needs_setup(di.ordinal, kSetupRouteTc)) {     // once per device
        IMX_CHECK_CUDA(cudaFuncSetAttribute(route_tc_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRtSmemMost));
        IMX_CHECK_CUDA(cudaFuncSetAttribute(route_tc_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRtSmemMost));
        IMX_CHECK_CUDA(cudaFuncSetAttribute(route_tc_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRtSmemMost));
        device_mark_setup(di.ordinal, kSetupRouteTc);
    }
    auto go = ceil_div(n, 32) <= di.sms ? launch_tile<32> : (ceil_div(n, 64) <= di.sms ? launch_tile<64> : launch_tile<128>);
    return go(x, n, H, Wr, logit_bias, E, k, norm, w_sg, topk_idx, topk_w, shared_gate, x16, order, status, stream);
}

}  // namespace imx
