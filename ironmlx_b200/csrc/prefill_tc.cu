// Host side of the tensor-core expert products (prefill_tc.cuh): which shapes and formats they take, the shared-memory plan,
// tensor maps and the launch.
#include <atomic>
#include <cstring>

#include "prefill_tc.h"

namespace imx {

using namespace prefill;

namespace {

std::atomic<int> g_spin_limit{kSpin};

int fmt_index(const QFormat& f) {
    if (f.mode == IMX_MODE_AFFINE) return f.bits == 4 ? FMT_A4 : (f.bits == 8 ? FMT_A8 : (f.bits == 2 ? FMT_A2 : -1));
    if (f.mode == IMX_MODE_MXFP8) return FMT_MXFP8;
    if (f.mode == IMX_MODE_NVFP4) return FMT_NVFP4;
    return -1;
}

// The two-term form of a format, or -1.
int two_term_index(const QFormat& f) {
    if (f.mode != IMX_MODE_AFFINE) return -1;
    return f.bits == 8 ? FMT_T8 : (f.bits >= 2 && f.bits <= 6 ? FMT_T2 + f.bits - 2 : -1);
}

int log2_exact(int v) {
    int l = 0;
    while ((1 << l) < v) ++l;
    return (1 << l) == v ? l : -1;
}

// bytes of one row of scales (K values) and the condition the copy engine puts on it
size_t scale_row(int K, const QFormat& f) { return (size_t)(K / f.group) * (f.mode == IMX_MODE_AFFINE ? 2 : 1); }
bool k_ok(int K, const QFormat& f) {
    if (K % kTileK || K % f.group) return false;
    const size_t sr = scale_row(K, f);
    return sr % 16 == 0 && K / f.group <= 256;
}
// ... and what the kernels themselves need of it (whole 32-bit words)
bool k_ok_any(int K, const QFormat& f) { return K % kTileK == 0 && K % f.group == 0 && scale_row(K, f) % 4 == 0 && K / f.group <= 256; }

// map of the packed codes of one stacked quantized matrix [rows, K]
int make_q_map(const QMat& m, size_t rows, int K, const QFormat& f, int fmt, CUtensorMap* w) {
    const int qrow = q_row_bytes(fmt);
    const size_t row_bytes = packed_row_bytes(K, f.bits);
    const int swz = qrow == 64 ? 64 : (qrow == 32 ? 32 : 0);
    IMX_TRY(make_tensor_map_2d(m.w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, rows, row_bytes, row_bytes, qrow, 64, false, w, false, swz));
    return IMX_OK;
}

// Shared memory of a launch: [panel][stages][two scale buffers][control block].  As many stages as fit,
// at most 8 (4 with two-term weights: the ring of A tiles in tensor memory has 256 columns) and, with a resident
// panel, at most the shortest reduction's K steps (the ring's back-pressure then also guards the panel).
bool make_plan(const QFormat& f, int fmt, int K_max, int K_min, bool wide, bool xr, bool ts, Plan* out, bool pair = false, int epi_row = 0) {
    const size_t q_tile = 128u * (size_t)q_row_bytes(fmt);
    const size_t sc = (size_t)128 * scale_row(K_max, f) * (f.mode == IMX_MODE_AFFINE ? 2 : 1);
    const size_t panel = xr ? (size_t)(K_max / kTileK) * kXBytes : 0;
    const size_t stage = (xr ? 0 : (size_t)kXBytes * (wide && !pair ? 2 : 1) + (ts ? 0 : kWBytes)) + q_tile;
    const size_t epi = wide ? (size_t)8 * 64 * (size_t)epi_row : 0;
    const size_t fixed = panel + 2 * sc + epi + sizeof(Bars) + 1024;
    if (fixed + 2 * stage > kSmemMost) return false;
    int st = (int)((kSmemMost - fixed) / stage);
    const int most = two_term(fmt) ? 4 : kMaxStages;
    if (st > most) st = most;
    if (xr && st > K_min / kTileK) st = K_min / kTileK;
    if (st < 2) return false;
    out->p = TcParams{};
    out->p.stages = st;
    out->p.stage_bytes = (int)stage;
    out->p.sc_bytes = (int)sc;
    out->p.panel_bytes = (int)panel;
    out->p.epi_bytes = (int)epi;
    out->p.spin_limit = g_spin_limit.load();
    out->p.lg_group = log2_exact(f.group);
    out->smem = fixed + (size_t)st * stage;
    out->wide = wide;
    out->pair = pair;
    out->xr = xr;
    return true;
}

// Wide tiles of one product: in pairs of CTAs where the weight tiles of a unit pair up, else one CTA each.  16-bit
// results are turned round in shared memory (first product 48, second 80 bytes a slot).
constexpr int kEpiFirst = 48, kEpiSecond = 80;
bool wide_plan(const QFormat& f, int fmt, int K_max, int K_min, bool even, int epi_row, Plan* out) {
    return (even && make_plan(f, fmt, K_max, K_min, true, false, true, out, true, epi_row)) ||
           make_plan(f, fmt, K_max, K_min, true, false, true, out, false, epi_row);
}

// Bytes a slot of the second product's transposing buffer: 16-bit rows without a factor per slot go through it to
// 16-byte stores, fp32 rows, rows with a factor (those of every two-term matrix) and rows that do not start on a
// multiple of 16 bytes leave as single values.
int second_epi(const void* rows16, bool scaled) { return rows16 != nullptr && !scaled && (uintptr_t)rows16 % 16 == 0 ? kEpiSecond : 0; }

}  // namespace

#ifdef IMX_TC_PROFILE
namespace prefill {
template <int FMT>
int read_prof(unsigned long long* out32);
}
extern "C" IMX_API int imx_debug_tc_prof(unsigned long long* out32) { return prefill::read_prof<prefill::FMT_A4>(out32); }
#endif

// Test hook (include/ironmlx_b200_testing.h).
void testing_prefill_give_up(int on) { g_spin_limit.store(on ? 0 : kSpin); }

static bool tc_supported(const ExpertSet& s, bool second_only, bool (*ok)(int, const QFormat&)) {
    const QFormat& f = s.fmt;
    if (fmt_index(f) < 0) return false;
    if (log2_exact(f.group) < 0 || f.group > 128 || f.group < 16) return false;
    if (f.mode == IMX_MODE_AFFINE && f.group < 32) return false;
    if (s.n_in % 128 || s.n_mid % 64) return false;
    // the second product alone never reduces over n_in (a plain quantized matmul with any number of output rows)
    if ((!second_only && !ok(s.n_in, f)) || !ok(s.n_mid, f)) return false;
    if (s.has_extra && (s.x_mid % 64 || !ok(s.x_mid, f))) return false;
    return true;
}
bool prefill_tc_supported(const ExpertSet& s, bool second_only) { return tc_supported(s, second_only, k_ok); }
bool tc_rows32_supported(const ExpertSet& s) {
    return (s.fmt.mode == IMX_MODE_MXFP8 || s.fmt.mode == IMX_MODE_NVFP4) && tc_supported(s, false, k_ok_any);
}

// Do the weight tiles of a unit pair up (64 gate and 64 up rows, 128 output rows a tile)?
static bool first_even(const ExpertSet& s) { return s.n_mid % 128 == 0 && (!s.has_extra || s.x_mid % 128 == 0); }
static bool second_even(const ExpertSet& s) { return s.n_in % 256 == 0; }

bool two_term_supported(const ExpertSet& s, bool second_only) {
    const QFormat& f = s.fmt;
    const int fmt = two_term_index(f);
    if (fmt < 0 || log2_exact(f.group) < 0 || f.group < 32 || f.group > 128) return false;
    if (s.n_in % 128 || (!second_only && s.n_mid % 64) || (s.has_extra && s.x_mid % 64)) return false;
    // packed rows advance in whole 16-byte pieces (the pitch a tiled copy needs)
    auto ok = [&](int K) { return k_ok_any(K, f) && packed_row_bytes(K, f.bits) % 16 == 0; };
    if ((!second_only && !ok(s.n_in)) || !ok(s.n_mid) || (s.has_extra && !ok(s.x_mid))) return false;
    const int mid_max = s.has_extra && s.x_mid > s.n_mid ? s.x_mid : s.n_mid;
    Plan p;
    return (second_only || wide_plan(f, fmt, s.n_in, s.n_in, first_even(s), kEpiFirst, &p)) &&
           wide_plan(f, fmt, mid_max, mid_max, second_even(s), second_epi(nullptr, true), &p);
}

// What the copy engine asks of the matrices' addresses (the other kernels take any 16 / 4-byte aligned tensor).
bool tc_aligned(const ExpertSet& s, bool second_only) {
    auto ok = [](const QMat& m) { return (((uintptr_t)m.w | (uintptr_t)m.scales | (uintptr_t)m.biases) % 16) == 0; };
    if (!ok(s.down) || (!second_only && !(ok(s.gate) && ok(s.up)))) return false;
    return !s.has_extra || (ok(s.x_down) && (second_only || (ok(s.x_gate) && ok(s.x_up))));
}

// variant: 0 = the shipped configuration (tensor-memory operand, 256-slot tiles in both products), 3 = the same with
// two-term weights, 1 = tensor-memory operand, 128-slot tiles and streamed activations everywhere, 2 = as 1 with the
// dequantized tile in shared memory (1, 2: cross-checks).
int launch_prefill_tc(const GroupedArgs& a, cudaStream_t stream, cudaEvent_t mid, int variant) {
    IMX_REQUIRE(variant == 3 ? two_term_supported(a.set, a.second_only != 0)
                : (variant == 0 && a.out16 == nullptr && tc_rows32_supported(a.set)) || prefill_tc_supported(a.set, a.second_only != 0),
                "prefill path: format/shape not supported");
    IMX_REQUIRE((a.row_index == nullptr || a.xs != nullptr || a.second_only) && a.n_slots > 0,
                "prefill path: slot-ordered activation buffer missing");
    IMX_REQUIRE(tc_aligned(a.set, a.second_only != 0), "prefill path: weights, scales and biases must be 16-byte aligned");
    if (a.max_units == 0) return IMX_OK;
    const ExpertSet& s = a.set;
    const QFormat& f = s.fmt;
    const int fmt = variant == 3 ? two_term_index(f) : fmt_index(f);
    const bool ts = variant != 2;
    const int x_mid = s.has_extra ? s.x_mid : s.n_mid;
    const int mid_max = s.n_mid > x_mid ? s.n_mid : x_mid;
    const int mid_min = s.n_mid < x_mid ? s.n_mid : x_mid;

    DeviceInfo di;
    IMX_TRY(current_device(&di));
    auto plan = [&](int K_max, int K_min, bool wide, bool xr, Plan* out) -> bool {
        return make_plan(f, fmt, K_max, K_min, wide, xr, ts, out);
    };
    Plan gu = {}, dn = {};
    IMX_REQUIRE(a.out16 == nullptr || a.row_scale == nullptr, "prefill path: fp16 rows carry no weight per slot");
    IMX_REQUIRE(a.out_bf16 == nullptr || (a.second_only && variant != 1 && variant != 2), "prefill path: bf16 rows belong to the second product alone");
    IMX_REQUIRE((uintptr_t)a.out16 % 16 == 0, "prefill path: fp16 rows must be 16-byte aligned");
    const int epi_second = second_epi(a.out_bf16 != nullptr ? (const void*)a.out_bf16 : a.out16, a.row_scale != nullptr);
    if (variant == 3) {
        IMX_REQUIRE((a.second_only || wide_plan(f, fmt, s.n_in, s.n_in, first_even(s), kEpiFirst, &gu)) &&
                        wide_plan(f, fmt, mid_max, mid_min, second_even(s), epi_second, &dn),
                    "two-term path: sizes exceed shared memory");
    } else {
        if (!a.second_only && !(variant == 0 && wide_plan(f, fmt, s.n_in, s.n_in, first_even(s), kEpiFirst, &gu)))
            IMX_REQUIRE(plan(s.n_in, s.n_in, false, false, &gu), "prefill path: sizes exceed shared memory");
        // second product: 256-slot tiles with streamed activations as well (c3: 276 us against 377 us with 128-slot
        // tiles and the activation panel resident, one CTA a tile); the resident panel where the wide stages do not fit
        if (!(variant == 0 && (wide_plan(f, fmt, mid_max, mid_min, second_even(s), epi_second, &dn) ||
                               (a.out_bf16 == nullptr && plan(mid_max, mid_min, false, true, &dn)))))
            IMX_REQUIRE(plan(mid_max, mid_min, false, false, &dn), "prefill path: sizes exceed shared memory");
    }
    gu.p.nt_r = s.n_mid / 64;
    gu.p.nt_x = x_mid / 64;
    dn.p.nt_r = dn.p.nt_x = s.n_in / 128;
    // the order of a block of 16 the first product's epilogue writes: the one the second product's weights are
    // unpacked in
    int order[16];
    expert_block_order(f, order);
    unsigned long long lut = 0;
    for (int pos = 0; pos < 16; ++pos) lut |= (unsigned long long)order[pos] << (4 * pos);
    gu.p.ord_lut = dn.p.ord_lut = lut;

    // activations in sorted-slot order (the `take_axis` of moe.rs:124-127, once for all experts)
    const __half* xsrc = a.in;                     // already slot-ordered when there is no row index
    if (a.row_index != nullptr && !a.second_only) {
        IMX_TRY(launch_gather_rows(a.in, a.row_index, a.n_slots, (size_t)s.n_in * 2, a.xs, stream, a.slots_end_dev, a.slots_resume));
        xsrc = a.xs;
    }
    TcMaps mgu, mdn;
    std::memset(&mgu, 0, sizeof(mgu));
    if (!a.second_only)
        IMX_TRY(make_tensor_map_2d(xsrc, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (size_t)a.n_slots, (size_t)s.n_in, (size_t)s.n_in * 2,
                                   kTileK, 128, true, &mgu.x));
    IMX_TRY(make_tensor_map_2d(a.act, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (size_t)a.n_slots, (size_t)mid_max, (size_t)a.act_stride * 2,
                               kTileK, 128, true, &mdn.x));
    // routed experts: gate and up rows live in one stacked matrix [E*2I, H]; down in [E*H, I]
    if (!a.second_only) IMX_TRY(make_q_map(s.gate, (size_t)s.num_experts * 2 * s.n_mid, s.n_in, f, fmt, &mgu.w[0]));
    IMX_TRY(make_q_map(s.down, (size_t)s.num_experts * s.n_in, s.n_mid, f, fmt, &mdn.w[0]));
    mgu.w[1] = mgu.w[2] = mgu.w[0];
    mdn.w[1] = mdn.w[0];
    if (s.has_extra) {
        if (!a.second_only) {
            IMX_TRY(make_q_map(s.x_gate, (size_t)s.x_mid, s.n_in, f, fmt, &mgu.w[1]));
            IMX_TRY(make_q_map(s.x_up, (size_t)s.x_mid, s.n_in, f, fmt, &mgu.w[2]));
        }
        IMX_TRY(make_q_map(s.x_down, (size_t)s.n_in, s.x_mid, f, fmt, &mdn.w[1]));
    }
    mdn.w[2] = mdn.w[1];

    // attributes of the format's kernels, once per device (the first call, outside any stream capture)
    const bool first = device_needs_setup(di.ordinal, kSetupPrefillTc + fmt);
    switch (fmt) {
        case FMT_A4: return launch_fmt<FMT_A4>(a, gu, dn, ts, mgu, mdn, di, first, stream, mid);
        case FMT_A8: return launch_fmt<FMT_A8>(a, gu, dn, ts, mgu, mdn, di, first, stream, mid);
        case FMT_A2: return launch_fmt<FMT_A2>(a, gu, dn, ts, mgu, mdn, di, first, stream, mid);
        case FMT_MXFP8: return launch_fmt<FMT_MXFP8>(a, gu, dn, ts, mgu, mdn, di, first, stream, mid);
        case FMT_NVFP4: return launch_fmt<FMT_NVFP4>(a, gu, dn, ts, mgu, mdn, di, first, stream, mid);
        case FMT_T2: return launch_fmt<FMT_T2>(a, gu, dn, ts, mgu, mdn, di, first, stream, mid);
        case FMT_T8: return launch_fmt<FMT_T8>(a, gu, dn, ts, mgu, mdn, di, first, stream, mid);
        case FMT_T3: return launch_fmt<FMT_T3>(a, gu, dn, ts, mgu, mdn, di, first, stream, mid);
        case FMT_T4: return launch_fmt<FMT_T4>(a, gu, dn, ts, mgu, mdn, di, first, stream, mid);
        case FMT_T5: return launch_fmt<FMT_T5>(a, gu, dn, ts, mgu, mdn, di, first, stream, mid);
        case FMT_T6: return launch_fmt<FMT_T6>(a, gu, dn, ts, mgu, mdn, di, first, stream, mid);
    }
    set_error("prefill path: unknown format");
    return IMX_ERR_INVALID;
}

}  // namespace imx
