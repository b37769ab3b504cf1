// Grouped expert products on the 5th-generation tensor cores, every weight format: affine 2/4/8-bit, mxfp8 and nvfp4 as one
// fp16 value a weight, affine 2/3/4/5/6/8-bit as the sum of two (TwoTerm below):
//
//   first product   act[slot, :] = silu(x W_gate^T) * (x W_up^T)       (moe.rs:26-30)
//   second product  out[slot, :] = row_scale[slot] * (act W_down^T)    (moe.rs:31, 155-161)
//
// each the grouped form of `quantized_matmul(transpose = true)` (mlx/src/nn/linear.rs:51-63), with `tcgen05.mma`
// (kind::f16, fp16 x fp16 -> fp32) and the accumulator in tensor memory.
//
// The WEIGHTS are the A operand (M = 128 weight rows, one tensor-memory lane each; 256 in a pair of CTAs), the sorted
// slots of one expert are the N side (the unit's rows rounded up to 16 or 32, at most 256), K in steps of 64.  The packed
// weights are dequantized by producer warps straight into TENSOR MEMORY (`tcgen05.st`), and the MMA takes A from there:
// the dequantized tile never passes through shared memory, which the 128 x 128 tile of an smem-smem MMA saturates.  Shared
// memory carries only what the copy engine brings: the activation tile (B operand, 128-byte swizzle) and the packed
// codes.  A variant with the dequantized tile in shared memory (TS = false) is kept as a cross-check.
//
// One persistent CTA per SM, 20 warps, specialised:
//   warp 0        issues the MMAs (one elected lane; of a pair, CTA 0's), commits a stage back to the loader and the
//                 finished accumulator to the epilogue
//   warp 1        allocates / frees tensor memory
//   warp 2        loader: tiled TMA copies of the activation tile and the packed codes (two boxes of 64 rows) per K step
//                 and, once per tile, the tile's scale (and bias) rows as runs of bytes
//   warps 4..7    epilogue, and 16..19 for the other half of a wide tile's slots (or the other accumulator): tcgen05.ld,
//                 16-bit rows turned round in shared memory and stored 16 bytes at a time.  First product: in every 16
//                 lanes eight hold gate rows and eight the matching up rows, so that a thread gets both values of a
//                 (row, slot) and SwiGLU needs no exchange
//   warps 8..15   producers, two groups of four warps on alternating K steps; a thread owns one weight row: its 16 to 64
//                 bytes of codes -> 64 fp16 values (or pairs of them) -> tcgen05.st of 32 columns (two-term: 64)
// Every wait is bounded; on expiry the CTA records a status, every role leaves its loop, what is in flight is waited for
// and tensor memory is freed.  Wide tiles run in clusters of two CTAs (PAIR below); no multicast loads.
//
// Scales: affine rounds s*q+b once to fp16 (two terms: to 22 bits).  nvfp4: q * (e4m3 block scale) is exact in fp16, the
// fp32 tensor scale is applied in the epilogue.  mxfp8: the e4m3 value times 2^(s - r), r the largest scale exponent of
// the weight row, is exact in fp16 (down to 2^-24 of the row's largest magnitude); 2^(r - 127) is applied per row in the
// epilogue.
#pragma once
#include <cuda.h>

#include <cstring>
#include <type_traits>

#include "decode_common.cuh"
#include "prefill_tc.h"
#include "tcgen05.cuh"

namespace imx {
namespace prefill {

using namespace decode;
using namespace tc;

// Per-role cycle counters of CTA 0, compiled in only for timing experiments (-DIMX_TC_PROFILE).
#ifdef IMX_TC_PROFILE
static __device__ unsigned long long g_tc_prof[2][16];
#define PROF_DECL long long _pt = 0, _p0 = clock64(), _pw[3] = {0, 0, 0};
#define PROF_BEGIN _pt = clock64();
#define PROF_END(i) _pw[i] += clock64() - _pt;
#define PROF_FLUSH(role)                                                                     \
    if (lane == 0 && blockIdx.x == 0) {                                                      \
        for (int _i = 0; _i < 3; ++_i) g_tc_prof[SWIGLU ? 1 : 0][(role) * 4 + _i] = _pw[_i]; \
        g_tc_prof[SWIGLU ? 1 : 0][(role) * 4 + 3] = clock64() - _p0;                         \
    }
#else
#define PROF_DECL
#define PROF_BEGIN
#define PROF_END(i)
#define PROF_FLUSH(role)
#endif

// Four (two) 8 x 8 matrices of 16-bit values in the MMA fragment layout (thread t: row t / 4, columns 2 (t % 4), + 1) to
// shared memory, transposed: lane 8 m + i names the 16 bytes column i of matrix m goes to.
__device__ __forceinline__ void stmatrix4_trans(uint32_t addr, uint32_t m0, uint32_t m1, uint32_t m2, uint32_t m3) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(m0), "r"(m1), "r"(m2), "r"(m3)
                 : "memory");
}
__device__ __forceinline__ void stmatrix2_trans(uint32_t addr, uint32_t m0, uint32_t m1) {
    asm volatile("stmatrix.sync.aligned.m8n8.x2.trans.shared.b16 [%0], {%1, %2};" ::"r"(addr), "r"(m0), "r"(m1) : "memory");
}
__device__ __forceinline__ void st_global_128(void* p, uint4 v) {
    asm volatile("st.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// `bytes` consecutive bytes (16-byte aligned, a multiple of 16) to shared memory.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
    return v;
}
// two fp32 -> packed fp16 (lo, hi), clamped to the finite range: one instruction
__device__ __forceinline__ uint32_t pack_f16_sat(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}
// silu with the approximate exponential and reciprocal (relative error ~1e-6, far inside the fp16 rounding that follows)
__device__ __forceinline__ float silu_fast(float g) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-1.4426950408889634f * g));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return g * r;
}
__device__ __forceinline__ void st_global_u16(void* p, uint32_t v) {
    asm volatile("st.global.u16 [%0], %1;" ::"l"(p), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ uint16_t ld_global_u16(const void* p) {
    uint16_t v;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
__device__ __forceinline__ __half2 bf16_to_half2(uint32_t b) {
    return __float2half2_rn(__uint_as_float(b << 16));
}

// A ring position: stage slot and phase of the n-th K step of the CTA.
struct Ring {
    int s;
    uint32_t ph;
    __device__ __forceinline__ void advance(int by, int stages) {
        s += by;
        while (s >= stages) {
            s -= stages;
            ph ^= 1u;
        }
    }
};

// What a tile is made of: one 128-row weight tile x (a part of) the sorted slots of one work unit.
struct TileInfo {
    int expert, slot0, rows, ntile, extra;
    int K;
    int first;              // first tile of its work item (XR: the activation panel is loaded with it)
};

// Walks this CTA's tiles.  Work units hold up to 256 slots.  SPLIT: the kernel's tiles take at most 128
// slots, so a larger unit is cut into two halves (multiples of 16 rows).  XR = false: a work item is one
// (unit part, weight tile), items dealt round-robin.  XR = true: a work item is a unit part with all its
// weight tiles in turn (its activation panel stays in shared memory).  nt_r / nt_x: weight tiles per unit of
// the routed experts / the extra expert.  body(tile, index) returns false to stop.
// PAIR: the two CTAs of a cluster take neighbouring weight tiles of the same unit (nt_r and nt_x are even).
template <bool SWIGLU, bool XR, bool SPLIT, bool PAIR, typename F>
__device__ __forceinline__ void for_each_tile(const GroupedArgs& a, int nt_r, int nt_x, F&& body) {
    const int rank = PAIR ? (int)(blockIdx.x & 1) : 0;
    if (PAIR) {
        nt_r >>= 1;
        nt_x >>= 1;
    }
    const int first = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, step = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    const int n_r = a.n_units[1], n_x = a.n_units[0] - n_r;
    const int tiles_r = n_r * nt_r;
    const int parts = SPLIT ? 2 : 1;
    const int total = (XR ? n_r + n_x : tiles_r + n_x * nt_x) * parts;
    int it = 0;
    for (int w0 = first; w0 < total; w0 += step) {
        const int part = SPLIT ? (w0 & 1) : 0;
        const int w = SPLIT ? (w0 >> 1) : w0;
        int unit, nt0, ntn = 1;
        if (XR) {
            unit = w;
            nt0 = 0;
            ntn = w < n_r ? nt_r : nt_x;
        } else if (w < tiles_r) {
            unit = w / nt_r;
            nt0 = w - unit * nt_r;
        } else {
            const int l = w - tiles_r;
            unit = n_r + l / nt_x;
            nt0 = l - (l / nt_x) * nt_x;
        }
        const WorkUnit u = a.units[unit];
        TileInfo t;
        t.expert = u.expert;
        t.slot0 = u.slot0;
        t.rows = u.rows;
        if (SPLIT) {
            const int h0 = u.rows <= 128 ? u.rows : (((u.rows + 1) >> 1) + 15) & ~15;
            if (part == 1) {
                t.slot0 = u.slot0 + h0;
                t.rows = u.rows - h0;
            } else {
                t.rows = h0;
            }
            if (t.rows <= 0) continue;
        }
        t.extra = u.expert >= a.set.num_experts;
        t.K = SWIGLU ? a.set.n_in : (t.extra ? a.set.x_mid : a.set.n_mid);
        for (int nt = nt0; nt < nt0 + ntn; ++nt, ++it) {
            t.ntile = PAIR ? 2 * nt + rank : nt;
            t.first = nt == nt0;
            if (!body(t, it)) return;
        }
    }
}

// Tensor-map index and first row of the two 64-row halves of 128-row weight tile `sub` of an expert.
template <bool SWIGLU>
__device__ __forceinline__ void tile_rows(const GroupedArgs& a, const TileInfo& t, int sub, int& mi0, int& mi1, int& row0, int& row1) {
    if (SWIGLU) {
        if (t.extra) { mi0 = 1; mi1 = 2; row0 = row1 = sub * 64; }
        else { mi0 = mi1 = 0; row0 = t.expert * 2 * a.set.n_mid + sub * 64; row1 = row0 + a.set.n_mid; }
    } else {
        mi0 = mi1 = t.extra ? 1 : 0;
        row0 = (t.extra ? 0 : t.expert * a.set.n_in) + sub * 128;
        row1 = row0 + 64;
    }
}

// Row of the 128-row tile (0..127: the order of the two TMA boxes: first product 64 gate rows, then the 64
// matching up rows) a tensor-memory lane holds.  First product: in every group of 16 lanes the first 8 hold
// gate rows and the other 8 the matching up rows, so that a 16-lane tensor-memory load hands a thread the gate
// and the up value of the same (row, slot) and SwiGLU needs no exchange between threads.  The 16 rows of two
// groups are a block of 16 output columns, taken in the order their values are stored in (ord_lut: the order the
// second product's weights are unpacked in), so that neighbouring lanes write neighbouring values.
template <bool SWIGLU>
__device__ __forceinline__ int tile_row_of_lane(int lane128, unsigned long long ord_lut) {
    if (!SWIGLU) return lane128;
    const int grp = lane128 >> 4, w = lane128 & 15;
    const int at = (grp & 1) * 8 + (w & 7);
    return ((w >> 3) << 6) + (grp >> 1) * 16 + (int)((ord_lut >> (4 * at)) & 0xf);
}

// ── dequantization of one weight row's K step: 64 values -> 32 registers of fp16 pairs ──
// q: shared address of the row's packed bytes (chunk c of 16 bytes at q + ((c ^ swz) << 4)).
template <int FMT>
struct Dequant;

template <>
struct Dequant<FMT_A4> {
    // scale/bias of a half step (32 values) given as half2 pairs
    static __device__ __forceinline__ void run(uint32_t q, uint32_t swz, const __half2 (&sc)[2], const __half2 (&bi)[2],
                                               uint32_t (&out)[32]) {
        const __half2 c1024 = __float2half2_rn(1024.f), c64 = __float2half2_rn(64.f);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const uint4 v4 = lds128(q + ((c ^ swz) << 4));
            const uint32_t words[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                // eight codes of a word -> (0,4) (1,5) (2,6) (3,7): the order the activation rows use
                uint32_t r[4];
                const uint32_t v = words[j], v8 = v >> 8;
                asm("lop3.b32 %0, %1, 0x000f000f, 0x64006400, 0xea;" : "=r"(r[0]) : "r"(v));
                asm("lop3.b32 %0, %1, 0x00f000f0, 0x54005400, 0xea;" : "=r"(r[1]) : "r"(v));
                asm("lop3.b32 %0, %1, 0x000f000f, 0x64006400, 0xea;" : "=r"(r[2]) : "r"(v8));
                asm("lop3.b32 %0, %1, 0x00f000f0, 0x54005400, 0xea;" : "=r"(r[3]) : "r"(v8));
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const __half2 qh = __hsub2(bits_h2(r[e]), (e & 1) ? c64 : c1024);      // exact code
                    out[(c * 4 + j) * 4 + e] = h2_bits(__hfma2(qh, sc[c], bi[c]));      // scale*q + bias
                }
            }
        }
    }
};

template <>
struct Dequant<FMT_A8> {
    static __device__ __forceinline__ void run(uint32_t q, uint32_t swz, const __half2 (&sc)[2], const __half2 (&bi)[2],
                                               uint32_t (&out)[32]) {
        const __half2 c1024 = __float2half2_rn(1024.f);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint4 v4 = lds128(q + ((c ^ swz) << 4));
            const uint32_t words[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                // four codes of a word -> (0,2) (1,3)
                uint32_t r0, r1;
                asm("prmt.b32 %0, %1, 0x64646464, 0x4240;" : "=r"(r0) : "r"(words[j]));
                asm("prmt.b32 %0, %1, 0x64646464, 0x4341;" : "=r"(r1) : "r"(words[j]));
                out[(c * 4 + j) * 2 + 0] = h2_bits(__hfma2(__hsub2(bits_h2(r0), c1024), sc[c >> 1], bi[c >> 1]));
                out[(c * 4 + j) * 2 + 1] = h2_bits(__hfma2(__hsub2(bits_h2(r1), c1024), sc[c >> 1], bi[c >> 1]));
            }
        }
    }
};

template <>
struct Dequant<FMT_A2> {
    static __device__ __forceinline__ void run(uint32_t q, uint32_t swz, const __half2 (&sc)[2], const __half2 (&bi)[2],
                                               uint32_t (&out)[32]) {
        (void)swz;
        const __half2 c1024 = __float2half2_rn(1024.f);
        const uint4 v4 = lds128(q);
        const uint32_t words[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            // sixteen codes of a word -> (J, J+8), J = 0..7
#pragma unroll
            for (int J = 0; J < 8; ++J) {
                uint32_t r;
                const uint32_t v = words[j] >> (2 * J);
                asm("lop3.b32 %0, %1, 0x00030003, 0x64006400, 0xea;" : "=r"(r) : "r"(v));
                out[j * 8 + J] = h2_bits(__hfma2(__hsub2(bits_h2(r), c1024), sc[j >> 1], bi[j >> 1]));
            }
        }
    }
};

template <>
struct Dequant<FMT_MXFP8> {
    // mult[h]: 2^(s - r) of the half step's group as a half2
    static __device__ __forceinline__ void run(uint32_t q, uint32_t swz, const __half2 (&mult)[2], const __half2 (&)[2],
                                               uint32_t (&out)[32]) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint4 v4 = lds128(q + ((c ^ swz) << 4));
            const uint32_t words[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t r0, r1;
                asm("{\n\t.reg .b16 lo, hi;\n\t"
                    "mov.b32 {lo, hi}, %2;\n\t"
                    "cvt.rn.f16x2.e4m3x2 %0, lo;\n\t"
                    "cvt.rn.f16x2.e4m3x2 %1, hi;\n\t}"
                    : "=r"(r0), "=r"(r1)
                    : "r"(words[j]));
                out[(c * 4 + j) * 2 + 0] = h2_bits(__hmul2(bits_h2(r0), mult[c >> 1]));
                out[(c * 4 + j) * 2 + 1] = h2_bits(__hmul2(bits_h2(r1), mult[c >> 1]));
            }
        }
    }
};

template <>
struct Dequant<FMT_NVFP4> {
    // sc4: the four e4m3 block scales of the step (one per 16 values), low byte first
    static __device__ __forceinline__ void run(uint32_t q, uint32_t swz, uint32_t sc4, uint32_t (&out)[32]) {
        uint32_t s01, s23;
        asm("{\n\t.reg .b16 lo, hi;\n\t"
            "mov.b32 {lo, hi}, %2;\n\t"
            "cvt.rn.f16x2.e4m3x2 %0, lo;\n\t"
            "cvt.rn.f16x2.e4m3x2 %1, hi;\n\t}"
            : "=r"(s01), "=r"(s23)
            : "r"(sc4));
        uint32_t sb[4];
        asm("prmt.b32 %0, %1, %1, 0x1010;" : "=r"(sb[0]) : "r"(s01));
        asm("prmt.b32 %0, %1, %1, 0x3232;" : "=r"(sb[1]) : "r"(s01));
        asm("prmt.b32 %0, %1, %1, 0x1010;" : "=r"(sb[2]) : "r"(s23));
        asm("prmt.b32 %0, %1, %1, 0x3232;" : "=r"(sb[3]) : "r"(s23));
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const uint4 v4 = lds128(q + ((c ^ swz) << 4));
            const uint32_t words[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                // a word = 8 values = half a block of 16: blocks 2c (j < 2) and 2c + 1
                uint32_t r[4];
                asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
                    "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
                    "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
                    "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
                    "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
                    "cvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                    : "r"(words[j]));
                const __half2 s = bits_h2(sb[2 * c + (j >> 1)]);
#pragma unroll
                for (int e = 0; e < 4; ++e) out[(c * 4 + j) * 4 + e] = h2_bits(__hmul2(bits_h2(r[e]), s));
            }
        }
    }
};

// ── two-term weights ────────────────────────────────────────────────────────
// The formats no 16-bit kernel serves (affine 3/5/6-bit, groups of 32) had their weights in fp32 in the scalar kernel, and
// the decode kernels keep affine weights exact.  One fp16 rounding of s * q + b would be a loss, so the MMA gets the weight
// as a sum of two fp16 terms, hi + lo, good to 22 bits, with two MMAs per 16 values: the tile of A is 64 tensor-memory
// columns per K step.  Everything is exact but the last rounding of lo:
//   p = rn(q * s), e = q * s - p           exact: q and s have 8 bits at most, what p (11 bits) leaves of 16 fits e
//   hi = rn(p + b), lo = rn(e + err)       err = the rounding error of p + b (Knuth's two-sum)
// fp16's range is met by a power of two 2^k per weight row, from the row's largest |s| 2^bits or |b|, taken back in
// the epilogue (fp32); scales below 2^-21 of that lose bits to fp16's subnormals, an absolute error of 2^-38 of the row's
// largest weight.  Infinite or NaN scales make the whole row NaN.  Error against fp64, 2-norm, two terms / scalar kernel:
// 2048 x 8192 6-bit, 100 rows 1.659308e-3 / 1.659305e-3 of the output, nearly all of it the rounding to bf16; fp32 rows
// of the expert stage 2.068e-4 / 2.067e-4, the fp16 SwiGLU rows' (what is more comes from the tensor cores' sums, which
// truncate: 7e-6).
// Measured on a B200 against the scalar kernels, 1000 tokens over 256 experts of 2048 x 512, 6-bit: both products 5.65 ms ->
// 0.48 ms (the block 5.73 -> 0.54 ms); what bounds it now is the dequantization: twelve half-precision operations a pair
// of values in eight warps, two thirds of a K step's time.  From one row on: 1 token 206 -> 83 us a block, a row through
// 2048 x 4096 86 -> 34 us.  Codes are pulled out in pairs (a, a + D) of a window of the bit stream, so that the second one
// lands in the upper half-word HS bits up (that factor goes into its copy of the scale); codes of a block of 16
// that have no partner at that distance pair with their neighbour.
template <int BITS>
struct TwoTerm {
    static constexpr int D = PairOrder<BITS>::D;
    static constexpr int HS = BITS * D - 16;                 // bit of the upper half-word the second code starts at
    __host__ __device__ static constexpr int first(int p) { return PairOrder<BITS>::first(p); }
    __host__ __device__ static constexpr int dist(int p) { return PairOrder<BITS>::dist(p); }
    // the pair as 1024 + q (lower half), 1024 + 2^HS q (upper half)
    template <int BIT, int DIST>
    static __device__ __forceinline__ uint32_t pair(const uint32_t* w) {
        constexpr uint32_t m = (1u << BITS) - 1u;
        constexpr int i = BIT >> 5, sh = BIT & 31, need = DIST * BITS + BITS;
        uint32_t v, r;
        if constexpr (sh + need <= 32) v = w[i] >> sh;
        else v = __funnelshift_r(w[i], w[i + 1], sh);
        if constexpr (DIST == D) {
            asm("lop3.b32 %0, %1, %2, 0x64006400, 0xea;" : "=r"(r) : "r"(v), "n"(m | (m << (16 + HS))));
        } else {
            const uint32_t u = v << (16 + HS - DIST * BITS);
            asm("lop3.b32 %0, %1, %2, 0x64006400, 0xea;" : "=r"(r) : "r"(v), "n"(m));
            asm("lop3.b32 %0, %1, %2, %0, 0xea;" : "+r"(r) : "r"(u), "n"(m << (16 + HS)));
        }
        return r;
    }
    // two blocks of 16 values of one group (block BLK of the 64 on): 16 registers of hi pairs, 16 of lo pairs
    template <int BLK, int P>
    static __device__ __forceinline__ void one(const uint32_t* w, __half2 s, __half2 b, uint32_t* hi_out, uint32_t* lo_out) {
        const __half2 q = __hsub2(bits_h2(pair<BLK * 16 * BITS + first(P) * BITS, dist(P)>(w)), __float2half2_rn(1024.f));
        const __half2 pr = __hmul2_rn(q, s);
        const __half2 hi = __hadd2_rn(pr, b);
        const __half2 bb = __hsub2_rn(hi, pr);
        __half2 lo = __hadd2_rn(__hsub2_rn(pr, __hsub2_rn(hi, bb)), __hsub2_rn(b, bb));
        if (BITS > 3) lo = __hadd2_rn(lo, __hfma2(q, s, __hneg2(pr)));   // 3 + 8 bits: the product is exact
        *hi_out = h2_bits(hi);
        *lo_out = h2_bits(lo);
    }
    template <int BLK>
    static __device__ __forceinline__ void block(const uint32_t* w, __half2 s, __half2 b, uint32_t* hi, uint32_t* lo) {
        one<BLK, 0>(w, s, b, hi + 0, lo + 0); one<BLK, 1>(w, s, b, hi + 1, lo + 1);
        one<BLK, 2>(w, s, b, hi + 2, lo + 2); one<BLK, 3>(w, s, b, hi + 3, lo + 3);
        one<BLK, 4>(w, s, b, hi + 4, lo + 4); one<BLK, 5>(w, s, b, hi + 5, lo + 5);
        one<BLK, 6>(w, s, b, hi + 6, lo + 6); one<BLK, 7>(w, s, b, hi + 7, lo + 7);
    }
};
__device__ __forceinline__ float pow2_f32(int e) {           // e in [-126, 127]
    return __uint_as_float((uint32_t)(e + 127) << 23);
}
// Running maximum over two scales (or biases) of a row as bf16 magnitudes, `up` added to the exponent of each.
__device__ __forceinline__ uint32_t max_mag(uint32_t v, uint32_t up, uint32_t m) { return __vmaxu2(m, (v & 0x7fff7fffu) + up); }
// f(word) for every 32-bit word of a row of scales (a multiple of 4 bytes), 16 bytes a load where the length allows.
template <typename F>
__device__ __forceinline__ void each_word_shared(uint32_t addr, uint32_t bytes, F&& f) {
    if (bytes % 16 == 0) {
        for (uint32_t i = 0; i < bytes; i += 16) {
            const uint4 v = lds128(addr + i);
            f(v.x); f(v.y); f(v.z); f(v.w);
        }
    } else {
        for (uint32_t i = 0; i < bytes; i += 4) f(lds32(addr + i));
    }
}
template <typename F>
__device__ __forceinline__ void each_word_global(const uint8_t* p, int bytes, F&& f) {
    if (bytes % 16 == 0) {
        for (int i = 0; i < bytes; i += 16) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(p + i));
            f(v.x); f(v.y); f(v.z); f(v.w);
        }
    } else {
        for (int i = 0; i < bytes; i += 4) f(__ldg(reinterpret_cast<const uint32_t*>(p + i)));
    }
}
// The exponent k of the row's power of two: its largest |s| 2^bits or |b| comes to lie in [2^13, 2^14).
__device__ __forceinline__ int row_shift(uint32_t mag2) { return 140 - (int)(max(mag2 & 0xffffu, mag2 >> 16) >> 7); }

// 2^d (d <= 0) as an fp16 bit pattern in both halves; below 2^-24 it is zero.
__device__ __forceinline__ __half2 pow2_half2(int d) {
    uint32_t b = 0;
    if (d >= -14) b = (uint32_t)(d + 15) << 10;
    else if (d >= -24) b = 1u << (d + 24);
    return bits_h2(b | (b << 16));
}

__device__ __forceinline__ uint32_t hmax_bytes(uint32_t m) {
    m = max(m & 0xffu, max((m >> 8) & 0xffu, max((m >> 16) & 0xffu, m >> 24)));
    return m;
}

// WIDE: tiles of up to 256 slots (N = 256 per MMA: the issue cost of a tcgen05.mma, about 110 cycles whatever
// its N, is then covered by the 128 cycles it runs) with one accumulator of 256 columns and eight epilogue
// warps; otherwise tiles of up to 128 slots and two accumulators, the epilogue of tile i overlapping the MMAs
// of tile i+1.  XR: the unit part's activation panel stays in shared memory for all its weight tiles.
// PAIR (wide tiles): two CTAs of a cluster share the activation tile.  Their weight tiles are neighbours, M = 256 in
// one `cta_group::2` MMA that CTA 0 issues; each CTA brings and keeps half of the tile's slots (16 instead of 32 KB
// a K step, so that eight stages fit instead of five) and dequantizes its own 128 weight rows.  CTA 0's full and
// acc_empty barriers collect both CTAs' arrivals, commits reach the empty and acc_full barriers of both.  Two CTAs on
// their own each read the whole activation tile from L2 and waited for it with five stages in flight; measured on a
// B200, both products: 8192 tokens over 256 experts of 2048 x 512, 4-bit 736 -> 580 us, 4096 tokens nvfp4 445 -> 356 us,
// 1777 tokens 8-bit 417 -> 328 us, 16384 skewed tokens 2-bit 1303 -> 1032 us.  What bounds them now is the MMAs (M = 256,
// N = 256: 128 cycles each, 512 of the 577 a K step takes in the first product) and the epilogue between tiles.
// BF16: the rows leave rounded to bf16 (the second product alone).  A kernel of its own, since the epilogue is short of
// registers: with the choice made at run time every call of the block lost 2 to 4 %.
template <bool SWIGLU, int FMT, bool TS, bool WIDE, bool XR, bool PAIR, bool BF16>
__device__ __forceinline__ void prefill_tc_body(const GroupedArgs& a, const TcParams& p, const TcMaps& maps) {
    static_assert(!PAIR || WIDE, "pairs of CTAs: wide tiles");
    static_assert(!WIDE || (TS && !XR), "wide tiles: tensor-memory operand, streamed activations");
    constexpr bool TWO = two_term(FMT);
    static_assert(!TWO || (TS && WIDE), "two-term weights: 256-slot tiles, tensor-memory operand");
    constexpr int ACOLS = TWO ? 64 : 32;                     // tensor-memory columns of one stage's A tile
    constexpr int TBITS = TWO ? two_term_bits(FMT) : 4;
    constexpr int QROW = q_row_bytes(FMT);
    constexpr int QBYTES = 128 * QROW;                       // packed codes of one 128-row tile per K step
    constexpr bool AFFINE = FMT == FMT_A4 || FMT == FMT_A8 || FMT == FMT_A2 || TWO;
    constexpr int XB = WIDE && !PAIR ? 2 * kXBytes : kXBytes;   // activation tile of a stage
    constexpr uint32_t Q_OFF = XR ? 0u : (uint32_t)(XB + (TS ? 0 : kWBytes));
    constexpr int NB = WIDE ? 1 : 2;                         // accumulator buffers
    constexpr int DCOLS = WIDE ? 256 : 128;                  // columns of one accumulator
    constexpr bool SPLIT = !WIDE;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    // [activation panel (XR)][stages][2 tiles' scale buffers][transposing buffers (WIDE)][control block]
    Bars* bars = reinterpret_cast<Bars*>(base + (size_t)p.panel_bytes + (size_t)p.stages * p.stage_bytes + 2 * (size_t)p.sc_bytes + p.epi_bytes);
    const uint32_t panel = smem_u32(base);
    const uint32_t sbase = panel + (uint32_t)p.panel_bytes;
    const uint32_t sc_base = sbase + (uint32_t)(p.stages * p.stage_bytes);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    volatile int* abort_flag = &bars->abort;
    const int stages = p.stages;

    if (tid == 0) {
        for (int s = 0; s < kMaxStages; ++s) {
            mbar_init(smem_u32(&bars->qfull[s]), 1);
            mbar_init(smem_u32(&bars->full[s]), PAIR ? 8 : 4);
            mbar_init(smem_u32(&bars->empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&bars->acc_full[b]), 1);
            mbar_init(smem_u32(&bars->acc_empty[b]), PAIR ? 16 : (WIDE ? 8 : 4));
            mbar_init(smem_u32(&bars->sfull[b]), 1);
            mbar_init(smem_u32(&bars->sempty[b]), 8);
        }
        mbar_init(smem_u32(&bars->retired), 1);
        bars->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)),
                         "r"(kTmemCols)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)),
                         "r"(kTmemCols)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync();                                // the peer's barriers are initialised before anyone arrives on them
    tc_fence_after();
    const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
    const uint32_t tmem = bars->tmem_base;

    if (warp == 0 && rank != 0) {
        // CTA 0 issues the pair's MMAs
    } else if (warp == 0) {
        // ── MMA issuer ──────────────────────────────────────────────────────
        Ring r = {0, 0u};
        PROF_DECL
        for_each_tile<SWIGLU, XR, SPLIT, PAIR>(a, p.nt_r, p.nt_x, [&](const TileInfo& t, int it) -> bool {
            const int buf = it % NB, round = it / NB;
            PROF_BEGIN
            if (!mbar_wait(smem_u32(&bars->acc_empty[buf]), (uint32_t)(round & 1) ^ 1u, abort_flag, p.spin_limit)) return false;
            PROF_END(0)
            tc_fence_after();
            const int ksteps = t.K / kTileK;
            const uint32_t idesc = PAIR ? idesc_for(256, (t.rows + 31) & ~31) : idesc_for(128, (t.rows + 15) & ~15);
            const uint32_t d = tmem + (uint32_t)(buf * DCOLS);
            for (int ks = 0; ks < ksteps; ++ks) {
                PROF_BEGIN
                if (!mbar_wait(smem_u32(&bars->full[r.s]), r.ph, abort_flag, p.spin_limit)) return false;
                PROF_END(1)
                tc_fence_after();
                PROF_BEGIN
                if (elect_one()) {
                    const uint32_t stage = sbase + (uint32_t)(r.s * p.stage_bytes);
                    const uint64_t dx = smem_desc(XR ? panel + (uint32_t)(ks * kXBytes) : stage);
#pragma unroll
                    for (int kk = 0; kk < kTileK / 16; ++kk) {
                        const uint32_t acc = (ks > 0 || kk > 0) ? 1u : 0u;
                        const uint32_t ta = tmem + kTmemA + (uint32_t)(r.s * ACOLS + kk * 8);
                        if (PAIR) umma_ts_pair(d, ta, dx + 2 * kk, idesc, acc);
                        else if (TS) umma_ts(d, ta, dx + 2 * kk, idesc, acc);
                        else umma_ss(d, smem_desc(stage + XB) + 2 * kk, dx + 2 * kk, idesc, acc);
                        if (TWO && PAIR) umma_ts_pair(d, ta + 32, dx + 2 * kk, idesc, 1u);
                        else if (TWO) umma_ts(d, ta + 32, dx + 2 * kk, idesc, 1u);
                    }
                    if (PAIR) {
                        umma_commit_pair(smem_u32(&bars->empty[r.s]));
                        if (ks == ksteps - 1) umma_commit_pair(smem_u32(&bars->acc_full[buf]));
                    } else {
                        umma_commit(smem_u32(&bars->empty[r.s]));            // stage free once these MMAs retire
                        if (ks == ksteps - 1) umma_commit(smem_u32(&bars->acc_full[buf]));
                    }
                }
                __syncwarp();
                PROF_END(2)
                r.advance(1, stages);
            }
            return true;
        });
        // nothing of this warp's is in flight when tensor memory is freed, also where a wait ran out
        if (elect_one()) {
            if (PAIR) umma_commit_own_pair(smem_u32(&bars->retired));
            else umma_commit(smem_u32(&bars->retired));
        }
        __syncwarp();
        mbar_drain(smem_u32(&bars->retired), 0u);
        PROF_FLUSH(0)
    } else if (warp == 2) {
        // ── loader (TMA): activation tile, packed codes, scales ─────────────
        Ring r = {0, 0u};
        int copied = 0, tiles = 0;                               // stages and tiles' scales this warp has started to copy
        PROF_DECL
        for_each_tile<SWIGLU, XR, SPLIT, PAIR>(a, p.nt_r, p.nt_x, [&](const TileInfo& t, int it) -> bool {
            const int ksteps = t.K / kTileK;
            int mi0, mi1, row0, row1;
            tile_rows<SWIGLU>(a, t, t.ntile, mi0, mi1, row0, row1);
            const int sbuf = it & 1;
            PROF_BEGIN
            if (!mbar_wait(smem_u32(&bars->sempty[sbuf]), (uint32_t)((it >> 1) & 1) ^ 1u, abort_flag, p.spin_limit)) return false;
            PROF_END(0)
            if (lane == 0) {
                // bytes of one row of scales for this reduction length
                const uint32_t srow = (uint32_t)(t.K >> p.lg_group) * (AFFINE ? 2u : 1u);
                const uint32_t bar = smem_u32(&bars->sfull[sbuf]);
                const uint32_t dst = sc_base + (uint32_t)(sbuf * p.sc_bytes);
                mbar_expect_tx(bar, (AFFINE ? 4u : 2u) * 64u * srow);
                // rows of scales lie one behind the other: 64 of them are one run of bytes, of any row length
                const ExpertSet& S = a.set;
                const QMat& m0 = SWIGLU ? (t.extra ? S.x_gate : S.gate) : (t.extra ? S.x_down : S.down);
                const QMat& m1 = SWIGLU ? (t.extra ? S.x_up : S.up) : m0;
                const size_t e_off = t.extra ? 0 : (size_t)t.expert * (SWIGLU ? S.gu_stride_s : S.dn_stride_s);
                const size_t r0 = e_off + (size_t)t.ntile * (SWIGLU ? 64 : 128) * srow, r1 = SWIGLU ? r0 : r0 + 64 * (size_t)srow;
                bulk_load(dst, m0.scales + r0, 64 * srow, bar);
                bulk_load(dst + 64 * srow, m1.scales + r1, 64 * srow, bar);
                if (AFFINE) {
                    bulk_load(dst + 128 * srow, m0.biases + r0, 64 * srow, bar);
                    bulk_load(dst + 192 * srow, m1.biases + r1, 64 * srow, bar);
                }
            }
            __syncwarp();
            ++tiles;
            // activation rows this tile needs: one box of 128 slots, a second one past 128 rows; of a pair, each
            // CTA brings its half of the slots
            const bool two = WIDE && !PAIR && t.rows > 128;
            const int xslot = t.slot0 + (PAIR ? (int)rank * (((t.rows + 31) & ~31) >> 1) : 0);
            for (int ks = 0; ks < ksteps; ++ks) {
                PROF_BEGIN
                if (!mbar_wait(smem_u32(&bars->empty[r.s]), r.ph ^ 1u, abort_flag, p.spin_limit)) return false;
                PROF_END(1)
                if (lane == 0) {
                    const uint32_t bar = smem_u32(&bars->qfull[r.s]);
                    const uint32_t stage = sbase + (uint32_t)(r.s * p.stage_bytes);
                    // XR: the panel's chunk ks is loaded with the part's first tile; the MMAs that read the
                    // previous part's chunk retired before this stage's slot came free (stages <= K steps)
                    const bool with_x = !XR || t.first;
                    mbar_expect_tx(bar, (uint32_t)(QBYTES + (with_x ? (two ? 2 * kXBytes : kXBytes) : 0)));
                    if (with_x) {
                        const uint32_t xdst = XR ? panel + (uint32_t)(ks * kXBytes) : stage;
                        tma_load_2d(xdst, &maps.x, ks * kTileK, xslot, bar);
                        if (two) tma_load_2d(xdst + kXBytes, &maps.x, ks * kTileK, t.slot0 + 128, bar);
                    }
                    tma_load_2d(stage + Q_OFF, &maps.w[mi0], q_step_byte(FMT, ks), row0, bar);
                    tma_load_2d(stage + Q_OFF + QBYTES / 2, &maps.w[mi1], q_step_byte(FMT, ks), row1, bar);
                }
                __syncwarp();
                r.advance(1, stages);
                ++copied;
            }
            return true;
        });
        // the copies still in flight where a wait ran out (else they were consumed long ago)
        for (int i = min(copied, stages); i > 0; --i) {
            if (--r.s < 0) {
                r.s = stages - 1;
                r.ph ^= 1u;
            }
            mbar_drain(smem_u32(&bars->qfull[r.s]), r.ph);
        }
        for (int it = max(0, tiles - 2); it < tiles; ++it) mbar_drain(smem_u32(&bars->sfull[it & 1]), (uint32_t)(it >> 1) & 1u);
        PROF_FLUSH(1)
    } else if ((warp >= 4 && warp < 8) || warp >= 16) {
        // ── epilogue ────────────────────────────────────────────────────────
        const int q = warp & 3;                                 // tensor-memory lane quarter
        const int eh = warp >= 16 ? 1 : 0;                      // WIDE: which half of the tile's slots; else: which accumulator
        const int lane128 = q * 32 + lane;
        // this warp's transposing buffer: 64 slots of 32 (second product: 64) bytes, rows padded so that eight of them
        // spread over all banks
        constexpr uint32_t kEpiRow = SWIGLU ? 48 : 80;
        const uint32_t ebuf = sc_base + 2u * (uint32_t)p.sc_bytes + (uint32_t)(eh * 4 + q) * 64u * kEpiRow;
        PROF_DECL
        for_each_tile<SWIGLU, XR, SPLIT, PAIR>(a, p.nt_r, p.nt_x, [&](const TileInfo& t, int it) -> bool {
            const int buf = it % NB, round = it / NB;
            if (!WIDE && buf != eh) return true;                    // two accumulators: one set of four warps each
            const ExpertSet& S = a.set;
            // Per-row output factors (before the accumulator is waited for: global loads): nvfp4's tensor scale,
            // mxfp8's 2^(largest scale exponent of the row - 127), two-term weights' 2^-k.
            auto row_factor = [&](const QMat& m, size_t estride, int r_in) -> float {
                if (TWO) {
                    const int srow = (t.K >> p.lg_group) * 2;
                    const size_t off = (t.extra ? 0 : (size_t)t.expert * estride) + (size_t)r_in * srow;
                    uint32_t mx = 0;
                    each_word_global(m.scales + off, srow, [&](uint32_t v) { mx = max_mag(v, (uint32_t)TBITS * 0x00800080u, mx); });
                    each_word_global(m.biases + off, srow, [&](uint32_t v) { mx = max_mag(v, 0u, mx); });
                    const int k = row_shift(mx);
                    return pow2_f32(-(k / 2)) * pow2_f32(-(k - k / 2));
                }
                if (AFFINE) return 1.f;
                if (FMT == FMT_NVFP4) return m.global_scale;
                const int srow = t.K >> 5;                          // one ue8m0 byte per 32 values
                const uint8_t* sp = m.scales + (t.extra ? 0 : (size_t)t.expert * estride) + (size_t)r_in * srow;
                uint32_t mx = 0;
                each_word_global(sp, srow, [&](uint32_t v) { mx = __vmaxu4(mx, v); });
                return ue8m0_to_f32(hmax_bytes(mx));
            };
            // [lane group of 16][gate, up], or the weight rows 16 gs + 8 r8 + lane / 4 of the warp's 32; second product
            // with one weight row a lane (fp32 rows): [0]
            float rf[4] = {1.f, 1.f, 1.f, 1.f};
            // rows that leave through the transposing buffer: the launch planned one (fp16 rows without a weight per slot
            // always have it; asked of the plan as well, their kernels came out 0.5 % slower)
            const bool frag_rows = !SWIGLU && WIDE && (BF16 ? p.epi_bytes != 0 : a.row_scale == nullptr && a.out16 != nullptr);
            if (SWIGLU) {
#pragma unroll
                for (int gs = 0; gs < 2; ++gs) {
                    const int idx = t.ntile * 64 + q * 16 + (int)((p.ord_lut >> (4 * (gs * 8 + (lane >> 2)))) & 0xf);
                    rf[2 * gs] = row_factor(t.extra ? S.x_gate : S.gate, S.gu_stride_s, idx);
                    rf[2 * gs + 1] = row_factor(t.extra ? S.x_up : S.up, S.gu_stride_s, idx);
                }
            } else if (frag_rows) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    rf[i] = row_factor(t.extra ? S.x_down : S.down, S.dn_stride_s, t.ntile * 128 + q * 32 + i * 8 + (lane >> 2));
            } else {
                rf[0] = row_factor(t.extra ? S.x_down : S.down, S.dn_stride_s, t.ntile * 128 + lane128);
            }
            PROF_BEGIN
            if (!mbar_wait(smem_u32(&bars->acc_full[buf]), (uint32_t)(round & 1), abort_flag, p.spin_limit)) return false;
            PROF_END(0)
            tc_fence_after();
            PROF_BEGIN
            float peak = 0.f;                                       // largest magnitude this thread rounds to fp16 in the tile
            const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * DCOLS);
            auto release = [&]() {                                  // all of this warp's TMEM reads are done
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (PAIR) mbar_arrive_cta0(smem_u32(&bars->acc_empty[buf]));
                    else mbar_arrive(smem_u32(&bars->acc_empty[buf]));
                }
            };
            if (SWIGLU) {
                // pieces of 64 slots x 16 lanes: 8 gate rows and the 8 matching up rows; a thread finishes row
                // lane/4 of the piece for the slots 8 j + 2 (lane % 4), +1
                const int n64 = (t.rows + 63) >> 6;
                const int c_lo = WIDE ? eh * 2 : 0, c_hi = WIDE ? min(n64, eh * 2 + 2) : n64;
                if (c_lo >= c_hi) release();
                // one piece: 64 slots from column 64 c on, lane group gs
                // (columns past the unit's rows hold what earlier tiles left: they are not counted as clamped)
                auto finish_piece = [&](int c, int gs, uint32_t (&o)[8]) {
                    const int n_ok = t.rows - c * 64 - 2 * (lane & 3);
                    uint32_t v[32];
                    tmem_ld_16x64(taddr + ((uint32_t)(gs * 16) << 16) + (uint32_t)(c * 64), v);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float g0 = __uint_as_float(v[4 * j]), g1 = __uint_as_float(v[4 * j + 1]);
                        float u0 = __uint_as_float(v[4 * j + 2]), u1 = __uint_as_float(v[4 * j + 3]);
                        if (!AFFINE || TWO) { g0 *= rf[2 * gs]; g1 *= rf[2 * gs]; u0 *= rf[2 * gs + 1]; u1 *= rf[2 * gs + 1]; }
                        const float r0 = silu_fast(g0) * u0, r1 = silu_fast(g1) * u1;
                        peak = fmaxf(peak, fmaxf(8 * j < n_ok ? fabsf(r0) : 0.f, 8 * j + 1 < n_ok ? fabsf(r1) : 0.f));
                        o[j] = pack_f16_sat(r0, r1);
                    }
                };
                const int pos0 = t.ntile * 64 + q * 16;                      // first of the warp's 16 stored columns
                auto store_piece = [&](int c, int gs, const uint32_t (&o)[8]) {
                    const int sl0 = c * 64 + 2 * (lane & 3);                 // first of this thread's slots
                    __half* dst = a.act + (size_t)(t.slot0 + sl0) * a.act_stride + pos0 + gs * 8 + (lane >> 2);
                    const int n_ok = t.rows - sl0;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        if (8 * j < n_ok) st_global_u16(dst + (size_t)(8 * j) * a.act_stride, o[j]);
                        if (8 * j + 1 < n_ok) st_global_u16(dst + (size_t)(8 * j + 1) * a.act_stride, o[j] >> 16);
                    }
                };
                if (WIDE) {
                    // everything leaves tensor memory before the first store: the accumulator is free that much earlier
                    uint32_t o[2][2][8];
#pragma unroll
                    for (int cc = 0; cc < 2; ++cc)
                        if (c_lo + cc < c_hi) {
                            finish_piece(c_lo + cc, 0, o[cc][0]);
                            finish_piece(c_lo + cc, 1, o[cc][1]);
                        }
                    if (c_lo < c_hi) release();
#pragma unroll
                    for (int cc = 0; cc < 2; ++cc)
                        if (c_lo + cc < c_hi) {
                            // 64 slots x 16 columns, turned round in shared memory: a slot's 32 bytes go out as two
                            // 16-byte stores, 16 slots at a time, instead of as single values
                            const uint32_t at = ebuf + (uint32_t)(lane & 7) * kEpiRow + (uint32_t)((lane >> 3) & 1) * 16u;
#pragma unroll
                            for (int j = 0; j < 8; ++j) stmatrix2_trans(at + (uint32_t)j * 8u * kEpiRow, o[cc][0][j], o[cc][1][j]);
                            __syncwarp();
                            const int sl0 = (c_lo + cc) * 64;
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const int sl = i * 16 + (lane >> 1);
                                const uint4 v = lds128(ebuf + (uint32_t)sl * kEpiRow + (uint32_t)(lane & 1) * 16u);
                                if (sl0 + sl < t.rows)
                                    st_global_128(a.act + (size_t)(t.slot0 + sl0 + sl) * a.act_stride + pos0 + (lane & 1) * 8, v);
                            }
                            __syncwarp();
                        }
                } else {
                    for (int c = c_lo; c < c_hi; ++c)
#pragma unroll
                        for (int gs = 0; gs < 2; ++gs) {
                            uint32_t o[8];
                            finish_piece(c, gs, o);
                            if (c == c_hi - 1 && gs == 1) release();
                            store_piece(c, gs, o);
                        }
                }
            } else {
                const int chunks = (t.rows + 31) >> 5;
                const int c_lo = WIDE ? eh * 4 : 0, c_hi = WIDE ? min(chunks, eh * 4 + 4) : chunks;
                if (c_lo >= c_hi) release();
                const int col = t.ntile * 128 + lane128;
                if (frag_rows && c_lo < c_hi) {
                    // All of the warp's columns leave tensor memory as packed pairs before the first is stored: the
                    // single accumulator is free for the next tile's MMAs that much earlier.  Then 64 slots x 32
                    // columns at a time are turned round in shared memory and go out as 16-byte pieces, 8 slots an
                    // instruction.  As single values, 64 bytes an instruction, the stores of a tile took longer than
                    // the MMAs of a 512-long reduction (role times of CTA 0, 8192 tokens: epilogue busy 274 of 357
                    // thousand cycles); the block went from 833 to 793 us.
                    const int n64 = (t.rows - eh * 128 + 63) >> 6;  // pieces of 64 slots of this warp's half: 1 or 2
                    // a piece as fragments: [8 weight rows][8 slots]
                    auto drain = [&](int c, uint32_t (&h)[4][8]) {
                        const int n_ok = t.rows - (eh * 2 + c) * 64 - 2 * (lane & 3);
#pragma unroll
                        for (int gs = 0; gs < 2; ++gs) {
                            uint32_t v[32];
                            tmem_ld_16x64(taddr + ((uint32_t)(gs * 16) << 16) + (uint32_t)((eh * 2 + c) * 64), v);
#pragma unroll
                            for (int j = 0; j < 8; ++j)
#pragma unroll
                                for (int r8 = 0; r8 < 2; ++r8) {
                                    float x0 = __uint_as_float(v[4 * j + 2 * r8]), x1 = __uint_as_float(v[4 * j + 2 * r8 + 1]);
                                    if (!AFFINE || TWO) { x0 *= rf[2 * gs + r8]; x1 *= rf[2 * gs + r8]; }
                                    if constexpr (BF16) {
                                        h[2 * gs + r8][j] = pack_bf16(x0, x1);
                                    } else {
                                        peak = fmaxf(peak, fmaxf(8 * j < n_ok ? fabsf(x0) : 0.f, 8 * j + 1 < n_ok ? fabsf(x1) : 0.f));
                                        h[2 * gs + r8][j] = pack_f16_sat(x0, x1);
                                    }
                                }
                        }
                    };
                    auto turn = [&](const uint32_t (&h)[4][8]) {
                        const uint32_t at = ebuf + (uint32_t)(lane & 7) * kEpiRow + (uint32_t)(lane >> 3) * 16u;
#pragma unroll
                        for (int j = 0; j < 8; ++j) stmatrix4_trans(at + (uint32_t)j * 8u * kEpiRow, h[0][j], h[1][j], h[2][j], h[3][j]);
                        __syncwarp();
                    };
                    auto flush = [&](int c) {
                        uint16_t* rows16 = BF16 ? reinterpret_cast<uint16_t*>(a.out_bf16) : reinterpret_cast<uint16_t*>(a.out16);
                        const int sl0 = (eh * 2 + c) * 64;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int sl = i * 8 + (lane >> 2);
                            const uint4 v = lds128(ebuf + (uint32_t)sl * kEpiRow + (uint32_t)(lane & 3) * 16u);
                            if (sl0 + sl < t.rows) {
                                const int slot = t.slot0 + sl0 + sl;
                                const int orow = a.out_index != nullptr ? a.out_index[slot] : slot;
                                st_global_128(rows16 + (size_t)orow * a.set.n_in + t.ntile * 128 + q * 32 + (lane & 3) * 8, v);
                            }
                        }
                        __syncwarp();
                    };
                    uint32_t h[4][8];
                    drain(0, h);
                    if (n64 == 1) release();
                    turn(h);
                    if (n64 > 1) {
                        drain(1, h);
                        release();
                    }
                    flush(0);
                    if (n64 > 1) {
                        turn(h);
                        flush(1);
                    }
                } else
                for (int c = c_lo; c < c_hi; ++c) {
                    uint32_t v[32];
                    tmem_ld32(taddr + c * 32, v);
                    if (c == c_hi - 1) release();
                    // the arithmetic first, for all 32 values and without a branch, then the stores under their
                    // row guards
                    float o[32];
                    uint32_t written = 0;                           // slots whose rows were written before this launch
                    if (a.row_scale != nullptr) {
                        // a weight per slot: one per lane, handed round by shuffle
                        const int my = c * 32 + lane;
                        // (the weight row's own factor, rf, belongs to the lane and is not handed round)
                        const float rs = my < t.rows ? a.row_scale[t.slot0 + my] : 1.f;
                        if (BF16 && TWO) written = __ballot_sync(0xffffffffu, rs != rs);
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            o[i] = (AFFINE && !TWO ? __uint_as_float(v[i]) : __uint_as_float(v[i]) * rf[0]) * __shfl_sync(0xffffffffu, rs, i);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = AFFINE && !TWO ? __uint_as_float(v[i]) : __uint_as_float(v[i]) * rf[0];
                    }
                    const size_t o0 = (size_t)(t.slot0 + c * 32) * a.set.n_in + col;
                    const int n_ok = t.rows - c * 32;
                    // (wide tiles: 16-bit rows without a weight per slot went out above)
                    if constexpr (BF16) {
                        __nv_bfloat16* y = a.out_bf16 + o0;
                        uint16_t kept[32];                          // (touched only where a row was written before)
                        if (TWO && written != 0)
                            for (uint32_t w = written; w != 0; w &= w - 1) {
                                const int i = __ffs(w) - 1;
                                kept[i] = ld_global_u16(y + (size_t)i * a.set.n_in);
                            }
#pragma unroll
                        for (int i = 0; i < 32; i += 2) {
                            const uint32_t h = pack_bf16(o[i], o[i + 1]);
                            if (i < n_ok) st_global_u16(y + (size_t)i * a.set.n_in, h);
                            if (i + 1 < n_ok) st_global_u16(y + (size_t)(i + 1) * a.set.n_in, h >> 16);
                        }
                        if (TWO && written != 0)
                            for (uint32_t w = written; w != 0; w &= w - 1) {
                                const int i = __ffs(w) - 1;
                                st_global_u16(y + (size_t)i * a.set.n_in, kept[i]);
                            }
                    } else if (!WIDE && a.out16 != nullptr && a.out_index != nullptr) {
                        // rows scattered to the positions the caller names (expert parallelism: straight into the
                        // buffer the rows travel back in): one index per lane, handed round by shuffle
                        const int my = c * 32 + lane;
                        const int orow = my < t.rows ? a.out_index[t.slot0 + my] : 0;
#pragma unroll
                        for (int i = 0; i < 32; i += 2) {
                            peak = fmaxf(peak, fmaxf(fabsf(o[i]), fabsf(o[i + 1])));
                            const uint32_t h = pack_f16_sat(o[i], o[i + 1]);
                            const int r0 = __shfl_sync(0xffffffffu, orow, i), r1 = __shfl_sync(0xffffffffu, orow, i + 1);
                            if (i < n_ok) st_global_u16(a.out16 + (size_t)r0 * a.set.n_in + col, h);
                            if (i + 1 < n_ok) st_global_u16(a.out16 + (size_t)r1 * a.set.n_in + col, h >> 16);
                        }
                    } else if (!WIDE && a.out16 != nullptr) {
#pragma unroll
                        for (int i = 0; i < 32; i += 2) {
                            peak = fmaxf(peak, fmaxf(fabsf(o[i]), fabsf(o[i + 1])));
                            const uint32_t h = pack_f16_sat(o[i], o[i + 1]);
                            if (i < n_ok) st_global_u16(a.out16 + o0 + (size_t)i * a.set.n_in, h);
                            if (i + 1 < n_ok) st_global_u16(a.out16 + o0 + (size_t)(i + 1) * a.set.n_in, h >> 16);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (i < n_ok) a.out[o0 + (size_t)i * a.set.n_in] = o[i];
                    }
                }
            }
            // values beyond the fp16 range were clamped: counted (per thread and tile), never silent
            if (peak > 65504.f && a.status != nullptr) atomicAdd(a.status + kStatusSaturations, 1);
            PROF_END(1)
            return true;
        });
        if (warp == 4) { PROF_FLUSH(2) }
    } else if (warp >= 8 && warp < 16) {
        // ── producers ───────────────────────────────────────────────────────
        // two groups of four warps on alternating K steps; a thread owns one weight row of the tile
        const int grp_id = (warp - 8) >> 2;
        const int lane128 = tid - 256 - grp_id * 128;     // tensor-memory lane = (warp % 4) * 32 + lane
        const int qrow = tile_row_of_lane<SWIGLU>(lane128, p.ord_lut);
        const uint32_t swz = QROW == 32 ? ((uint32_t)qrow >> 2) & 1u : (QROW == 64 ? ((uint32_t)qrow >> 1) & 3u : 0u);
        const uint32_t q_off = Q_OFF + (uint32_t)qrow * QROW;
        const uint32_t t_lane = tmem + ((uint32_t)((warp & 3) * 32) << 16) + kTmemA;
        // TS = false: this row's 128 bytes of the K-major swizzled weight tile
        const uint32_t w_off = (uint32_t)XB + (uint32_t)((lane128 >> 3) * 1024 + (lane128 & 7) * 128);
        Ring r = {0, 0u};
        r.advance(grp_id, stages);
        PROF_DECL
        for_each_tile<SWIGLU, XR, SPLIT, PAIR>(a, p.nt_r, p.nt_x, [&](const TileInfo& t, int it) -> bool {
            const int ksteps = t.K / kTileK;
            const int sbuf = it & 1;
            const uint32_t srow = (uint32_t)(t.K >> p.lg_group) * (AFFINE ? 2u : 1u);
            const uint32_t s_addr = sc_base + (uint32_t)(sbuf * p.sc_bytes) + (uint32_t)qrow * srow;
            const uint32_t b_addr = s_addr + 128u * srow;
            PROF_BEGIN
            if (!mbar_wait(smem_u32(&bars->sfull[sbuf]), (uint32_t)((it >> 1) & 1), abort_flag, p.spin_limit)) return false;
            PROF_END(0)
            int r_exp = 0;
            if (FMT == FMT_MXFP8) {
                uint32_t mx = 0;
                each_word_shared(s_addr, srow, [&](uint32_t v) { mx = __vmaxu4(mx, v); });
                r_exp = (int)hmax_bytes(mx);
            }
            float up0 = 1.f, up1 = 1.f;               // two-term weights: the row's 2^k, as two factors in fp32's range
            if (TWO) {
                uint32_t mx = 0;
                each_word_shared(s_addr, srow, [&](uint32_t v) { mx = max_mag(v, (uint32_t)TBITS * 0x00800080u, mx); });
                each_word_shared(b_addr, srow, [&](uint32_t v) { mx = max_mag(v, 0u, mx); });
                const int k = row_shift(mx);
                up0 = pow2_f32(k / 2);
                up1 = pow2_f32(k - k / 2);
            }
            int ks = grp_id;
            for (; ks < ksteps; ks += 2) {
                PROF_BEGIN
                if (!mbar_wait(smem_u32(&bars->qfull[r.s]), r.ph, abort_flag, p.spin_limit)) return false;
                PROF_END(1)
                PROF_BEGIN
                const uint32_t stage = sbase + (uint32_t)(r.s * p.stage_bytes);
                uint32_t out[32];
                if constexpr (TWO) {
                    using Tt = TwoTerm<TBITS>;
                    // the step's 64 codes of this row as a bit stream
                    uint32_t w[2 * TBITS];
                    if (TBITS % 2 == 0) {
#pragma unroll
                        for (int c = 0; c < TBITS / 2; ++c) {
                            const uint4 v = lds128(stage + q_off + (((uint32_t)c ^ (TBITS == 4 || TBITS == 8 ? swz : 0u)) << 4));
                            w[4 * c] = v.x; w[4 * c + 1] = v.y; w[4 * c + 2] = v.z; w[4 * c + 3] = v.w;
                        }
                    } else {
                        const uint32_t at = stage + q_off + (uint32_t)(ks & 1) * 8u;   // 24 ks or 40 ks, less the box's start
#pragma unroll
                        for (int c = 0; c < TBITS; ++c) {
                            const uint2 v = lds64(at + 8u * c);
                            w[2 * c] = v.x; w[2 * c + 1] = v.y;
                        }
                    }
                    const uint32_t ta = t_lane + (uint32_t)(r.s * ACOLS);
                    auto half_step = [&](auto hc) {
                        constexpr int h = decltype(hc)::value;
                        const uint32_t gi = (uint32_t)(ks * kTileK + h * 32) >> p.lg_group;
                        const float sf = __uint_as_float(lds16(s_addr + gi * 2) << 16) * up0 * up1;
                        const float bf = __uint_as_float(lds16(b_addr + gi * 2) << 16) * up0 * up1;
                        const __half2 s2 = __floats2half2_rn(sf, sf * (1.f / (float)(1 << Tt::HS)));
                        const __half2 b2 = __float2half2_rn(bf);
                        uint32_t hi[16], lo[16];
                        Tt::template block<2 * h>(w, s2, b2, hi, lo);
                        Tt::template block<2 * h + 1>(w, s2, b2, hi + 8, lo + 8);
                        tmem_st16(ta + 16u * h, hi);
                        tmem_st16(ta + 32u + 16u * h, lo);
                    };
                    half_step(std::integral_constant<int, 0>{});
                    half_step(std::integral_constant<int, 1>{});
                } else if constexpr (AFFINE) {
                    __half2 sc[2], bi[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t gi = (uint32_t)(ks * kTileK + h * 32) >> p.lg_group;
                        sc[h] = bf16_to_half2(lds16(s_addr + gi * 2));
                        bi[h] = bf16_to_half2(lds16(b_addr + gi * 2));
                    }
                    if (FMT == FMT_A4) Dequant<FMT_A4>::run(stage + q_off, swz, sc, bi, out);
                    if (FMT == FMT_A8) Dequant<FMT_A8>::run(stage + q_off, swz, sc, bi, out);
                    if (FMT == FMT_A2) Dequant<FMT_A2>::run(stage + q_off, swz, sc, bi, out);
                } else if constexpr (FMT == FMT_MXFP8) {
                    const uint32_t s2 = lds16(s_addr + (uint32_t)ks * 2);
                    __half2 mult[2] = {pow2_half2((int)(s2 & 0xffu) - r_exp), pow2_half2((int)(s2 >> 8) - r_exp)};
                    Dequant<FMT_MXFP8>::run(stage + q_off, swz, mult, mult, out);
                } else {
                    Dequant<FMT_NVFP4>::run(stage + q_off, swz, lds32(s_addr + (uint32_t)ks * 4), out);
                }
                if constexpr (TWO) {
                    tmem_st_wait();
                    tc_fence_before();
                } else if constexpr (TS) {
                    tmem_st32(t_lane + (uint32_t)(r.s * 32), out);
                    tc_fence_before();
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint32_t dst = stage + w_off + (((uint32_t)j ^ (uint32_t)(lane128 & 7)) << 4);
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(out[4 * j]), "r"(out[4 * j + 1]),
                                     "r"(out[4 * j + 2]), "r"(out[4 * j + 3])
                                     : "memory");
                    }
                    fence_async_proxy();                 // generic-proxy writes -> visible to the tensor-core reads
                }
                __syncwarp();
                if (lane == 0) {
                    if (PAIR) mbar_arrive_cta0(smem_u32(&bars->full[r.s]));
                    else mbar_arrive(smem_u32(&bars->full[r.s]));
                }
                PROF_END(2)
                r.advance(2, stages);
            }
            // the ring position is now `ks` steps into this tile; this group's next step is `grp_id` steps
            // into the next one
            const int delta = ksteps + grp_id - ks;       // -1, 0 or 1
            if (delta > 0) r.advance(delta, stages);
            else if (delta < 0) r.advance(2 * stages + delta, stages);   // one step back: two turns minus one
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->sempty[sbuf]));   // this warp is done with the tile's scales
            return true;
        });
        if (warp == 8) { PROF_FLUSH(3) }
    }

    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync();                                // neither CTA leaves while the other may arrive on its barriers
    if (warp == 1) {
        if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
    if (tid == 0 && bars->abort && a.status != nullptr) atomicExch(a.status, 3);
}

template <bool SWIGLU, int FMT, bool TS, bool WIDE, bool XR, bool BF16 = false>
__global__ void __launch_bounds__(kThreadsTc, 1)
prefill_tc_kernel(const GroupedArgs a, const TcParams p, const __grid_constant__ TcMaps maps) {
    prefill_tc_body<SWIGLU, FMT, TS, WIDE, XR, false, BF16>(a, p, maps);
}

template <bool SWIGLU, int FMT, bool BF16 = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreadsTc, 1)
prefill_pair_kernel(const GroupedArgs a, const TcParams p, const __grid_constant__ TcMaps maps) {
    prefill_tc_body<SWIGLU, FMT, true, true, false, true, BF16>(a, p, maps);
}

template <int FMT>
int configure() {
    constexpr int kSmem = (int)kSmemMost;
    IMX_CHECK_CUDA(cudaFuncSetAttribute(prefill_pair_kernel<true, FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    IMX_CHECK_CUDA(cudaFuncSetAttribute(prefill_pair_kernel<false, FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    IMX_CHECK_CUDA(cudaFuncSetAttribute(prefill_pair_kernel<false, FMT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    IMX_CHECK_CUDA(cudaFuncSetAttribute(prefill_tc_kernel<false, FMT, true, true, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    if constexpr (two_term(FMT)) {
        IMX_CHECK_CUDA(cudaFuncSetAttribute(prefill_tc_kernel<true, FMT, true, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        IMX_CHECK_CUDA(cudaFuncSetAttribute(prefill_tc_kernel<false, FMT, true, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        return IMX_OK;
    } else {
        IMX_CHECK_CUDA(cudaFuncSetAttribute(prefill_tc_kernel<false, FMT, true, false, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        IMX_CHECK_CUDA(cudaFuncSetAttribute(prefill_tc_kernel<true, FMT, true, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        IMX_CHECK_CUDA(cudaFuncSetAttribute(prefill_tc_kernel<true, FMT, true, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        IMX_CHECK_CUDA(cudaFuncSetAttribute(prefill_tc_kernel<false, FMT, true, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        IMX_CHECK_CUDA(cudaFuncSetAttribute(prefill_tc_kernel<false, FMT, true, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        IMX_CHECK_CUDA(cudaFuncSetAttribute(prefill_tc_kernel<false, FMT, true, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        IMX_CHECK_CUDA(cudaFuncSetAttribute(prefill_tc_kernel<true, FMT, false, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        IMX_CHECK_CUDA(cudaFuncSetAttribute(prefill_tc_kernel<false, FMT, false, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        return IMX_OK;
    }
}

template <int FMT>
int launch_fmt(const GroupedArgs& a, const Plan& gu, const Plan& dn, bool ts, const TcMaps& mgu, const TcMaps& mdn, const DeviceInfo& di,
               bool first, cudaStream_t stream, cudaEvent_t mid) {
    const int sms = di.sms;
    if (first) {
        IMX_TRY(configure<FMT>());
        device_mark_setup(di.ordinal, kSetupPrefillTc + FMT);
    }
    if (a.out_bf16 != nullptr) {
        if (dn.pair) prefill_pair_kernel<false, FMT, true><<<sms & ~1, kThreadsTc, dn.smem, stream>>>(a, dn.p, mdn);
        else if (dn.wide) prefill_tc_kernel<false, FMT, true, true, false, true><<<sms, kThreadsTc, dn.smem, stream>>>(a, dn.p, mdn);
        else if constexpr (!two_term(FMT))
            prefill_tc_kernel<false, FMT, true, false, false, true><<<sms, kThreadsTc, dn.smem, stream>>>(a, dn.p, mdn);
        IMX_LAUNCHED();
        IMX_CHECK_CUDA(cudaGetLastError());
        return IMX_OK;
    }
    if constexpr (two_term(FMT)) {
        if (!a.second_only) {
            if (gu.pair) prefill_pair_kernel<true, FMT><<<sms & ~1, kThreadsTc, gu.smem, stream>>>(a, gu.p, mgu);
            else prefill_tc_kernel<true, FMT, true, true, false><<<sms, kThreadsTc, gu.smem, stream>>>(a, gu.p, mgu);
            IMX_LAUNCHED();
            IMX_CHECK_CUDA(cudaGetLastError());
        }
        if (mid) IMX_CHECK_CUDA(cudaEventRecord(mid, stream));
        if (dn.pair) prefill_pair_kernel<false, FMT><<<sms & ~1, kThreadsTc, dn.smem, stream>>>(a, dn.p, mdn);
        else prefill_tc_kernel<false, FMT, true, true, false><<<sms, kThreadsTc, dn.smem, stream>>>(a, dn.p, mdn);
        IMX_LAUNCHED();
        IMX_CHECK_CUDA(cudaGetLastError());
        return IMX_OK;
    } else {
        if (!a.second_only) {
            if (gu.pair) prefill_pair_kernel<true, FMT><<<sms & ~1, kThreadsTc, gu.smem, stream>>>(a, gu.p, mgu);
            else if (!ts) prefill_tc_kernel<true, FMT, false, false, false><<<sms, kThreadsTc, gu.smem, stream>>>(a, gu.p, mgu);
            else if (gu.wide) prefill_tc_kernel<true, FMT, true, true, false><<<sms, kThreadsTc, gu.smem, stream>>>(a, gu.p, mgu);
            else prefill_tc_kernel<true, FMT, true, false, false><<<sms, kThreadsTc, gu.smem, stream>>>(a, gu.p, mgu);
            IMX_LAUNCHED();
            IMX_CHECK_CUDA(cudaGetLastError());
        }
        if (mid) IMX_CHECK_CUDA(cudaEventRecord(mid, stream));
        if (dn.pair) prefill_pair_kernel<false, FMT><<<sms & ~1, kThreadsTc, dn.smem, stream>>>(a, dn.p, mdn);
        else if (!ts) prefill_tc_kernel<false, FMT, false, false, false><<<sms, kThreadsTc, dn.smem, stream>>>(a, dn.p, mdn);
        else if (dn.wide) prefill_tc_kernel<false, FMT, true, true, false><<<sms, kThreadsTc, dn.smem, stream>>>(a, dn.p, mdn);
        else if (dn.xr) prefill_tc_kernel<false, FMT, true, false, true><<<sms, kThreadsTc, dn.smem, stream>>>(a, dn.p, mdn);
        else prefill_tc_kernel<false, FMT, true, false, false><<<sms, kThreadsTc, dn.smem, stream>>>(a, dn.p, mdn);
        IMX_LAUNCHED();
        IMX_CHECK_CUDA(cudaGetLastError());
        return IMX_OK;
    }
}

#ifdef IMX_TC_PROFILE
template <int FMT>
int read_prof(unsigned long long* out32) {
    return cudaMemcpyFromSymbol(out32, g_tc_prof, sizeof(unsigned long long) * 32) == cudaSuccess ? 0 : 2;
}
#endif

// The one instantiation of a format's kernels.
#ifdef IMX_TC_PROFILE
#define IMX_TC_FORMAT(F)                                    \
    template decltype(launch_fmt<F>) launch_fmt<F>;         \
    template decltype(read_prof<F>) read_prof<F>;
#else
#define IMX_TC_FORMAT(F) template decltype(launch_fmt<F>) launch_fmt<F>;
#endif

}  // namespace prefill
}  // namespace imx
