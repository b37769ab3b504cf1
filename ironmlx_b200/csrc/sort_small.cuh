// The one-block dispatch sort and its pieces (a kernel of its own in sort.cu, the tail of the decode-size router in
// route.cu).
#pragma once
#include "internal.h"

namespace imx {

// Block-wide exclusive scan of one int per thread (all threads must call).
static __device__ int block_exclusive_scan(int v, int* s_warp /*[32]*/, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        int w = (lane < (int)(blockDim.x >> 5)) ? s_warp[lane] : 0;
        int winc = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int t = __shfl_up_sync(0xffffffffu, winc, o);
            if (lane >= o) winc += t;
        }
        s_warp[lane] = winc - w;   // exclusive warp base
        if (lane == 31) s_warp[32] = winc;
    }
    __syncthreads();
    int res = s_warp[warp] + inc - v;
    if (total) *total = s_warp[32];
    __syncthreads();
    return res;
}

// Exclusive scan of s_tot[0..E) into offsets[0..E] (E <= blockDim).
static __device__ void scan_experts(const int* s_tot, int E, int32_t* __restrict__ offsets, int* s_off,
                             int* s_warp) {
    const int tid = threadIdx.x;
    int v = tid < E ? s_tot[tid] : 0;
    int total;
    int ex = block_exclusive_scan(v, s_warp, &total);
    if (tid < E) {
        s_off[tid] = ex;
        offsets[tid] = ex;
    }
    if (tid == 0) {
        s_off[E] = total;
        offsets[E] = total;
    }
    __syncthreads();
}

// Units of an expert with `cnt` rows.  Tensor-core tiles (unit sizes of 64 rows and more) cost the same
// whether full or not, so an expert that needs nu of them gets nu even parts (multiples of 16 rows) instead of
// full units and a remainder; very long lists (nu > 8, e.g. the shared expert's) keep the fixed stride.
__device__ __forceinline__ int unit_stride(int cnt, int ur, int nu) {
    if (ur < 64 || nu <= 1 || nu > 8) return ur;
    return (((cnt + nu - 1) / nu) + 15) & ~15;
}

struct SortAux {
    // optional extras emitted by the fused kernel (all may be null)
    const float* topk_w;     // [A] routing weight per flat assignment
    int top_k;
    int32_t* tok_of_slot;    // [A (+N)] token id per sorted slot
    float* w_of_slot;        // [A (+N)] routing weight per sorted slot
    const float* shared_gate;// [N] or null: appended after the A routed slots
    int n_tokens;
    int shared_token0;       // first of the n_tokens tokens the shared expert serves (0 unless tokens are sharded)
    WorkUnit* units;         // work units of `unit_rows` rows
    int32_t* n_units;
    int unit_rows;
    int32_t* sched;          // scheduler words to clear
    int sched_ints;
};

template <int THREADS>
__device__ void emit_aux(const SortAux& aux, const int32_t* __restrict__ perm, const int* s_off,
                         int E, int A, int* s_warp) {
    const int tid = threadIdx.x;
    if (aux.sched != nullptr)
        for (int i = tid; i < aux.sched_ints; i += THREADS) aux.sched[i] = 0;
    if (aux.tok_of_slot != nullptr) {
        const int total = s_off[E];
        for (int j = tid; j < total; j += THREADS) {
            int f = perm[j];
            aux.tok_of_slot[j] = f / aux.top_k;
            if (aux.w_of_slot) aux.w_of_slot[j] = aux.topk_w ? aux.topk_w[f] : 1.f;
        }
        if (aux.shared_gate != nullptr) {
            for (int t = tid; t < aux.n_tokens; t += THREADS) {
                aux.tok_of_slot[A + t] = aux.shared_token0 + t;
                if (aux.w_of_slot) aux.w_of_slot[A + t] = aux.shared_gate[aux.shared_token0 + t];
            }
        }
    }
    if (aux.units != nullptr) {
        const int ur = aux.unit_rows;
        // E routed experts + (optionally) the shared expert as pseudo-expert E
        const bool has_shared = aux.shared_gate != nullptr;
        int cnt = 0, pos0 = 0;
        if (tid < E) {
            cnt = s_off[tid + 1] - s_off[tid];
            pos0 = s_off[tid];
        } else if (tid == E && has_shared) {
            cnt = aux.n_tokens;
            pos0 = A;
        }
        int nu = (cnt + ur - 1) / ur;
        int total;
        int base = block_exclusive_scan(nu, s_warp, &total);
        const int per = unit_stride(cnt, ur, nu);
        for (int c = 0; c < nu; ++c) {
            WorkUnit u;
            u.expert = tid;
            u.slot0 = pos0 + c * per;
            u.rows = min(per, cnt - c * per);
            u.pad = 0;
            aux.units[base + c] = u;
        }
        if (tid == 0) aux.n_units[0] = total;
        if (tid == E) aux.n_units[1] = base;       // units of the routed experts (the extra expert's follow)
    }
}

// One block, at most kSmallSortIters ids per thread (A <= kSmallSortIters * THREADS, E <= kSmallSortExperts < THREADS):
// ids are read once, ranks stay in registers, and every output is written once (decode-size batches).  A warp owns a
// contiguous run of ids, so ranks follow the index order.  s_mem: small_sort_ints(THREADS / 32, E) ints.
constexpr int kSmallSortExperts = 256;
constexpr int kSmallSortIters = 4;
__host__ __device__ constexpr size_t small_sort_ints(int warps, int E) { return (size_t)warps * E + E + E + 1 + 33; }

template <int THREADS>
__device__ void sort_small_block(const int32_t* ids, int A, int E, int32_t* __restrict__ counts, int32_t* __restrict__ offsets,
                                 int32_t* __restrict__ perm, int32_t* __restrict__ inv_perm, const SortAux& aux, int* s_mem) {
    constexpr int WARPS = THREADS / 32;
    int* s_hist = s_mem;                       // [WARPS][E]
    int* s_tot = s_hist + WARPS * E;      // [E]
    int* s_off = s_tot + E;                    // [E+1]
    int* s_warp = s_off + E + 1;               // [33]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int per_warp = ((A + WARPS - 1) / WARPS + 31) & ~31;      // <= 32 * kSmallSortIters
    const int w_lo = warp * per_warp, w_hi = min(A, w_lo + per_warp);
    int e[kSmallSortIters], rank[kSmallSortIters];
    float w[kSmallSortIters];
#pragma unroll
    for (int it = 0; it < kSmallSortIters; ++it) {
        const int i = w_lo + it * 32 + lane;
        const bool in = it * 32 < per_warp && i < w_hi;
        int v = in ? __ldcg(ids + i) : -1;
        if (v < 0 || v >= E) v = -1;                      // moe.rs:100: out-of-range ids are dropped
        e[it] = v;
        w[it] = (in && aux.topk_w != nullptr) ? __ldcg(aux.topk_w + i) : 1.f;
        rank[it] = 0;
    }
    for (int i = tid; i < WARPS * E; i += THREADS) s_hist[i] = 0;
    __syncthreads();
    int* my_hist = s_hist + warp * E;
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int it = 0; it < kSmallSortIters; ++it) {
        if (it * 32 < per_warp) {
            // rank among equal ids: those of earlier passes of the warp, then lower lanes of this pass
            const unsigned peers = __match_any_sync(0xffffffffu, e[it]);
            const int before = e[it] >= 0 ? my_hist[e[it]] : 0;
            __syncwarp();
            if (e[it] >= 0) {
                const int r = __popc(peers & lt);
                if (r == 0) my_hist[e[it]] = before + __popc(peers);
                rank[it] = before + r;
            }
            __syncwarp();
        }
    }
    __syncthreads();
    for (int x = tid; x < E; x += THREADS) {          // exclusive scan over warps, per expert
        int run = 0;
        for (int v = 0; v < WARPS; ++v) {
            const int c = s_hist[v * E + x];
            s_hist[v * E + x] = run;
            run += c;
        }
        s_tot[x] = run;
        if (counts != nullptr) counts[x] = run;
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kSmallSortIters; ++it)
        if (e[it] >= 0) rank[it] += my_hist[e[it]];
    scan_experts(s_tot, E, offsets, s_off, s_warp);
#pragma unroll
    for (int it = 0; it < kSmallSortIters; ++it) {
        const int i = w_lo + it * 32 + lane;
        if (it * 32 < per_warp && i < w_hi) {
            if (e[it] >= 0) {
                const int pos = s_off[e[it]] + rank[it];
                perm[pos] = i;
                inv_perm[i] = pos;
                if (aux.tok_of_slot != nullptr) {
                    aux.tok_of_slot[pos] = i / aux.top_k;
                    if (aux.w_of_slot) aux.w_of_slot[pos] = w[it];
                }
            } else {
                inv_perm[i] = -1;
            }
        }
    }
    if (aux.tok_of_slot != nullptr && aux.shared_gate != nullptr) {
        for (int t = tid; t < aux.n_tokens; t += THREADS) {
            aux.tok_of_slot[A + t] = aux.shared_token0 + t;
            if (aux.w_of_slot) aux.w_of_slot[A + t] = __ldcg(aux.shared_gate + aux.shared_token0 + t);
        }
    }
    SortAux rest = aux;
    rest.tok_of_slot = nullptr;                           // written above; what remains: unit list, scheduler reset
    emit_aux<THREADS>(rest, nullptr, s_off, E, A, s_warp);
}

inline SortAux make_sort_aux(const SortExtras* ex) {
    SortAux aux = {};
    if (ex == nullptr) return aux;
    aux.topk_w = ex->topk_w;
    aux.top_k = ex->top_k > 0 ? ex->top_k : 1;
    aux.tok_of_slot = ex->tok_of_slot;
    aux.w_of_slot = ex->w_of_slot;
    aux.shared_gate = ex->shared_gate;
    aux.n_tokens = ex->n_tokens;
    aux.shared_token0 = ex->shared_token0;
    aux.units = ex->units;
    aux.n_units = ex->n_units;
    aux.unit_rows = ex->unit_rows > 0 ? ex->unit_rows : 8;
    aux.sched = ex->sched;
    aux.sched_ints = ex->sched_ints;
    return aux;
}

}  // namespace imx
