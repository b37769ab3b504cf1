// The tensor-core expert products (prefill_tc.cuh) as their host side sees them: formats, shared-memory layout and
// parameters of a launch.
#pragma once
#include <cuda.h>

#include "internal.h"

namespace imx {
namespace prefill {

constexpr int kTileK = 64;
constexpr int kXBytes = 128 * kTileK * 2;          // activation tile, 16 KB
constexpr int kWBytes = 128 * kTileK * 2;          // dequantized weight tile (TS = false only), 16 KB
constexpr int kMaxStages = 8;
constexpr uint32_t kTmemCols = 512;                // two 128-column accumulators + the ring of A tiles
constexpr uint32_t kTmemA = 256;                   // first column of the A ring (32 columns per stage)
constexpr int kThreadsTc = 640;                    // 20 warps: 4 control, 4 + 4 epilogue, 8 producers

// FMT_T*: affine weights as a two-term fp16 sum (hi + lo), see TwoTerm in prefill_tc.cuh.
enum { FMT_A4 = 0, FMT_A8 = 1, FMT_A2 = 2, FMT_MXFP8 = 3, FMT_NVFP4 = 4,
       FMT_T2 = 5, FMT_T3 = 6, FMT_T4 = 7, FMT_T5 = 8, FMT_T6 = 9, FMT_T8 = 10 };
__host__ __device__ constexpr bool two_term(int fmt) { return fmt >= FMT_T2; }
__host__ __device__ constexpr int two_term_bits(int fmt) { return fmt == FMT_T8 ? 8 : fmt - FMT_T2 + 2; }
// Bytes of one row the copy engine brings per K step of 64 values.  3- and 5-bit rows advance by 24 and 40 bytes a
// step and a copy starts on a multiple of 16: the box starts at the multiple below and is wide enough for both
// positions.  48-byte rows spread eight lanes' 16-byte loads over all banks without a swizzle.
__host__ __device__ constexpr int q_row_bytes(int fmt) {
    if (fmt == FMT_A8 || fmt == FMT_MXFP8 || fmt == FMT_T8) return 64;
    if (fmt == FMT_A2 || fmt == FMT_T2) return 16;
    return fmt == FMT_T3 || fmt == FMT_T5 || fmt == FMT_T6 ? 48 : 32;
}
// First byte of K step ks's box in a packed row (a multiple of 16).
__host__ __device__ constexpr int q_step_byte(int fmt, int ks) {
    return fmt == FMT_T3 ? (ks * 24) & ~15 : (fmt == FMT_T5 ? (ks * 40) & ~15 : ks * q_row_bytes(fmt));
}

struct Bars {                                      // shared-memory control block
    uint64_t qfull[kMaxStages];                    // activation tile + packed codes landed (TMA bytes)
    uint64_t full[kMaxStages];                     // weights of the stage dequantized
    uint64_t empty[kMaxStages];                    // MMAs that read the stage retired
    uint64_t acc_full[2];
    uint64_t acc_empty[2];
    uint64_t sfull[2];                             // scales of a tile landed
    uint64_t sempty[2];                            // ... and were consumed by all producer warps
    uint64_t retired;                              // the MMA warp's last commit
    uint32_t tmem_base;
    int abort;
};

struct TcMaps {
    CUtensorMap x;                                 // slot-ordered activations
    CUtensorMap w[3];                              // packed codes: [0] stacked routed matrix, [1]/[2] the extra expert's
};

struct TcParams {
    int nt_r, nt_x;                                // weight-row tiles per unit: routed / extra expert
    int stages;
    int stage_bytes;
    int sc_bytes;                                  // one tile's scale buffer
    int panel_bytes;                               // resident activation panel (0: streamed per stage)
    int lg_group;                                  // log2 of the group size
    int spin_limit;                                // bound of every wait
    int epi_bytes;                                 // wide tiles: the epilogue warps' transposing buffers
    unsigned long long ord_lut;                    // reduction index at position p of a block of 16, 4 bits each
};

constexpr size_t kSmemMost = 227 * 1024;

struct Plan {
    TcParams p;
    size_t smem;
    bool wide;
    bool pair;
    bool xr;
};

// Launches both products (or the second alone) of one weight format; `first` sets the kernels' attributes.  Each
// format is a translation unit of its own (prefill_tc_*.cu): the first call of a process then loads the kernels of its
// own format alone (one module of all: 29 ms, this: 4 ms).
template <int FMT>
int launch_fmt(const GroupedArgs& a, const Plan& gu, const Plan& dn, bool ts, const TcMaps& mgu, const TcMaps& mdn, const DeviceInfo& di,
               bool first, cudaStream_t stream, cudaEvent_t mid);

}  // namespace prefill
}  // namespace imx
