// Pieces of the router shared by its kernels: the fp16 copy's block orders and conversion, softmax and top-k of a warp.
#pragma once
#include "decode_common.cuh"

namespace imx {
namespace route {

// Block order of the fp16 copy by code width (0: rows stay as they are): position p of a block of 16 takes
// value order16<BITS>(p) of the source block.
template <int BITS>
__host__ __device__ constexpr int order16(int p) {
    if constexpr (BITS == 0) return p;
    else return decode::Codec<BITS>::order(p);
}
// Which of them `order` is, or -1.
inline int order_bits(const Order16& order) {
    const int widths[6] = {0, 4, 8, 2, 3, 6};           // (5-bit rows have the 4-bit order)
    for (int w = 0; w < 6; ++w) {
        bool same = true;
        for (int i = 0; i < 16; ++i) {
            const int want[6] = {order16<0>(i), order16<4>(i), order16<8>(i), order16<2>(i), order16<3>(i), order16<6>(i)};
            same = same && order.o[i] == want[w];
        }
        if (same) return widths[w];
    }
    return -1;
}
// One block of 16 bf16 values -> fp16 in block order BITS, pairs 1 and 3 of every 8 stored values times sc_odd:
// two 16-byte loads, the permutation in registers, two 16-byte stores.  SAT: values beyond fp16's range are clamped.
// Returns the sum of the 16 values as stored, the odd pairs scaled back, in stored order.
template <int BITS, bool SAT = true>
__device__ __forceinline__ float convert_block16(const __nv_bfloat16* __restrict__ src, __half* __restrict__ dst, float sc_odd,
                                                 float up0 = 1.f, float up1 = 1.f) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(src)), b = __ldg(reinterpret_cast<const uint4*>(src) + 1);
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    float in[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        in[2 * i] = __uint_as_float(w[i] << 16);
        in[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
    uint32_t o[8];
    float sum = 0.f;
    const float back = 1.f / sc_odd;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const float sc = (q & 1) ? sc_odd : 1.f;
        const float v0 = in[order16<BITS>(2 * q)] * sc * up0 * up1, v1 = in[order16<BITS>(2 * q + 1)] * sc * up0 * up1;
        const __half2 h = SAT ? __halves2half2(f32_to_f16_sat(v0), f32_to_f16_sat(v1)) : __floats2half2_rn(v0, v1);
        const float2 f = __half22float2(h);
        sum += (q & 1) ? f.x * back : f.x;
        sum += (q & 1) ? f.y * back : f.y;
        o[q] = *reinterpret_cast<const uint32_t*>(&h);
    }
    reinterpret_cast<uint4*>(dst)[0] = make_uint4(o[0], o[1], o[2], o[3]);
    reinterpret_cast<uint4*>(dst)[1] = make_uint4(o[4], o[5], o[6], o[7]);
    return sum;
}
template <bool SAT = true>
__device__ __forceinline__ float convert_block16(int obits, const __nv_bfloat16* __restrict__ src, __half* __restrict__ dst,
                                                 float sc_odd, float up0 = 1.f, float up1 = 1.f) {
    switch (obits) {
        case 4: return convert_block16<4, SAT>(src, dst, sc_odd, up0, up1);
        case 8: return convert_block16<8, SAT>(src, dst, sc_odd, up0, up1);
        case 2: return convert_block16<2, SAT>(src, dst, sc_odd, up0, up1);
        case 3: return convert_block16<3, SAT>(src, dst, sc_odd, up0, up1);
        case 6: return convert_block16<6, SAT>(src, dst, sc_odd, up0, up1);
        default: return convert_block16<0, SAT>(src, dst, sc_odd, up0, up1);
    }
}


template <int JMAX>
__device__ void softmax_topk_warp(const float* s_logits, int E, int k, bool norm, int32_t* out_idx,
                                  float* out_w) {
    const int lane = threadIdx.x & 31;
    float p[JMAX];
    float m = -INFINITY;
#pragma unroll
    for (int j = 0; j < JMAX; ++j) {
        int e = lane + 32 * j;
        p[j] = e < E ? s_logits[e] : -INFINITY;
        m = fmaxf(m, p[j]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < JMAX; ++j) {
        int e = lane + 32 * j;
        p[j] = e < E ? expf(p[j] - m) : 0.f;
        s += p[j];
    }
    s = warp_sum(s);
#pragma unroll
    for (int j = 0; j < JMAX; ++j) {
        int e = lane + 32 * j;
        p[j] = e < E ? p[j] / s : -1.f;   // -1 marks "not selectable"
    }
    float my_w = 0.f;
    int my_i = 0;
    float wsum = 0.f;
    // every lane keeps the best of its own candidates (lowest id first among equals); a round is then two
    // warp reductions (largest probability, lowest id that has it) and a rescan in the winning lane only.
    // Probabilities are >= 0 and the "taken" mark is -1, so the int view of the floats orders them.
    float bv;
    int bj;
    auto rescan = [&]() {
        bv = -1.f;
        bj = 0;
#pragma unroll
        for (int j = 0; j < JMAX; ++j) {
            if (p[j] > bv) {
                bv = p[j];
                bj = j;
            }
        }
    };
    rescan();
    for (int r = 0; r < k; ++r) {
        const int mine = __float_as_int(bv);
        const int top = __reduce_max_sync(0xffffffffu, mine);
        const int win = __reduce_min_sync(0xffffffffu, mine == top ? lane + 32 * bj : 0x7fffffff);
        const float wv = __int_as_float(top);
        if (mine == top && lane + 32 * bj == win) {
#pragma unroll
            for (int j = 0; j < JMAX; ++j)
                if (j == bj) p[j] = -1.f;
            rescan();
        }
        if (lane == (r & 31)) {
            my_w = wv;
            my_i = win;
        }
        wsum += wv;
        if ((r & 31) == 31 || r == k - 1) {      // flush up to 32 results
            int slot = (r & ~31) + lane;
            if (slot <= r) {
                out_idx[slot] = my_i;
                out_w[slot] = my_w;               // normalised below
            }
        }
    }
    __syncwarp();
    if (norm) {
        for (int slot = lane; slot < k; slot += 32) out_w[slot] = out_w[slot] / wsum;
    }
}

}  // namespace route
}  // namespace imx
