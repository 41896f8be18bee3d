// mpx_window.cuh -- gates applied in windows of up to 64, sector by sector over an active subset of the store
// (sm_100a).
//
// Two properties of a run of consecutive gates are used.
//   * Most terms of a truncated propagation are small: a term whose |c| cannot pass the lower_atol gate of any
//     gate of the window emits nothing there, and unless an emitting term's partner is it, all the window does
//     to it is multiply it by the cos of the gates it anticommutes with. On the 100-qubit circuit 98.6 % of the
//     anticommuting (term, gate) pairs are of that kind, and reading and writing those coefficients gate by
//     gate (scattered 32-byte sectors, 6.5e9 of them) was most of the propagation.
//   * A gate couples a term M only to M^G. Over the window every term therefore stays in its coset of the
//     group that the window's generators span, and cosets do not interact. A linear map f of the keys to 32
//     bits with f(G) = 0 for every generator of the window is constant on cosets; its hash deals the active
//     terms out to sectors, one thread block each, and a block runs all gates of the window on its sector with
//     block barriers only: no grid-wide synchronisation, no launch per gate, and no wait for the slowest block
//     at every gate. Longer windows spread the cost of the dense pass, shorter ones split the store into more
//     cosets; k_window_sample measures the sectors' loads for four lengths and the window takes the best, or
//     none where gate by gate takes less time (choose_length).
// One window is
//   k_window_close   one dense pass: the previous window's pending cos factors for its passive terms (in gate
//                    order, so every coefficient is rounded as gate-by-gate scaling rounds it), its counters,
//                    and the candidates of the next window (|c| times its largest |sin| above lower_atol);
//   k_window_sample  the sectors' loads for four window lengths, from a sample of the candidates;
//   k_window_count   each candidate's gate mask and sector for the best length;
//   k_window_scatter the sectors' lists (values, masks, terms), contiguous chunks;
//   k_window_gates   per sector and gate: the anticommuting active terms (one bit per list slot), cos scaling,
//                    lower_atol gate, structural cutoff, phase, partner lookup; then the leader/follower rule
//                    and the rotation of the pair or the append of the missing partner. A partner that is still
//                    passive first gets its pending cos factors and joins the list;
//   k_window_commit  the lists' values back to the store, and the bit-columns of the appends.
// Values live in the lists while the gates run, so a window whose appends do not fit changes nothing: the host
// grows the store and runs the window again. The per-gate semantics are those of Scan.h:193-396,
// Engine.h:364-513 and FusedApply.h:32-83; within a coset the gates run in order.
#pragma once

#include <cstdint>

#include "mpx_window.h"

namespace mpx {

// max(a, b), NaN once either is NaN (a gate whose |sin| is NaN lets every term emit)
__device__ __forceinline__ double max_or_nan(double a, double b) { return (b > a || b != b) ? b : a; }

template <int W>
__device__ __forceinline__ void load_key_l2(const uint64_t *keys, uint64_t i, uint64_t (&k)[W]) {
    const uint64_t *p = keys + i * W;
    if constexpr (W % 2 == 0) {
#pragma unroll
        for (int w = 0; w < W; w += 2) {
            const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2 *>(p + w));
            k[w] = v.x;
            k[w + 1] = v.y;
        }
    }
    else {
#pragma unroll
        for (int w = 0; w < W; ++w) k[w] = __ldcg(reinterpret_cast<const unsigned long long *>(p + w));
    }
}

// ----- the dense pass between two windows -------------------------------------------------------------------

// The linear tables of the window of K gates from step lo on, by one block: each key bit's gates, and for every
// window length its value of f. The generators (rows) are reduced to a basis in which every vector has a pivot
// bit that no other holds; every key bit gets a pseudo-random value of f, and then the pivots theirs so that f
// vanishes on the basis.
struct TableWork {
    uint64_t rows[kWindow][kMaxWords], mask[64 * kMaxWords];
    uint32_t inv[64 * kMaxWords];
    int pivot[kWindow];
    uint64_t odd;
};
__device__ __forceinline__ void window_tables(const GateDesc *__restrict__ gates, uint32_t L, uint32_t lo, int K, int W,
                                              WindowTables &t, uint64_t *comm, TableWork &s) {
    const int tid = static_cast<int>(threadIdx.x), T = static_cast<int>(blockDim.x);
    for (int k = tid; k < kWindow * W; k += T) {
        const int j = k / W, w = k % W;
        s.rows[j][w] = j < K ? gates[L - 1 - (lo + j)].g[w] : 0ull;
    }
    for (int c = tid; c < 64 * W; c += T) {
        uint64_t m = 0;
#pragma unroll 16
        for (int j = 0; j < K; ++j) m |= ((gates[L - 1 - (lo + j)].fold[c / 64] >> (c % 64)) & 1ull) << j;
        s.mask[c] = m;
        t.mask[c] = m;
    }
    if (tid < kWindow) {
        t.sin[tid] = tid < K ? gates[L - 1 - (lo + tid)].abs_sin : 0.0;
        s.pivot[tid] = -1;
    }
    if (tid < 32) {
        const uint32_t o0 = __ballot_sync(0xFFFFFFFFu, tid < K && gates[L - 1 - (lo + tid)].g_odd != 0);
        const uint32_t o1 = __ballot_sync(0xFFFFFFFFu, tid + 32 < K && gates[L - 1 - (lo + tid + 32)].g_odd != 0);
        if (tid == 0) t.odd = s.odd = o0 | (static_cast<uint64_t>(o1) << 32);
    }
    __syncthreads();
    if (tid < K) { // the gates' own anticommutation
        uint64_t mask = 0;
        int pop = 0;
        for (int w = 0; w < W; ++w) {
            pop += __popcll(s.rows[tid][w]);
            for (uint64_t x = s.rows[tid][w]; x != 0; x &= x - 1) mask ^= s.mask[64 * w + __ffsll(static_cast<long long>(x)) - 1];
        }
        comm[tid] = (pop & 1) ? mask ^ s.odd : mask;
    }
    __syncthreads();
    const int r = tid % kWindow; // row r, words tid / kWindow, ...
    int i = 0;
    for (int len = 0; len < kLengths; ++len) {
        for (const int end = static_cast<int>(window_length(len, K)); i < end; ++i) {
            int p = -1;
            for (int w = 0; w < W && p < 0; ++w)
                if (s.rows[i][w] != 0) p = 64 * w + __ffsll(static_cast<long long>(s.rows[i][w])) - 1;
            const bool has = p >= 0 && r != i && ((s.rows[r][p >> 6] >> (p & 63)) & 1ull) != 0;
            __syncthreads();
            if (has)
                for (int w = tid / kWindow; w < W; w += T / kWindow) s.rows[r][w] ^= s.rows[i][w];
            if (tid == 0) s.pivot[i] = p;
            __syncthreads();
        }
        for (int c = tid; c < 64 * W; c += T) s.inv[c] = static_cast<uint32_t>(mix64(static_cast<uint64_t>(c) * 0x9E3779B97F4A7C15ull + 1));
        __syncthreads();
        uint32_t f = 0;
        const int pv = tid < kWindow ? s.pivot[tid] : -1;
        if (pv >= 0)
            for (int w = 0; w < W; ++w)
                for (uint64_t x = s.rows[tid][w]; x != 0; x &= x - 1) {
                    const int c = 64 * w + __ffsll(static_cast<long long>(x)) - 1;
                    if (c != pv) f ^= s.inv[c];
                }
        __syncthreads();
        if (pv >= 0) s.inv[pv] = f;
        __syncthreads();
        for (int c = tid; c < 64 * W; c += T) t.inv[len][c] = s.inv[c];
        __syncthreads();
    }
}

constexpr int kCloseWarps = 8;
constexpr int kCloseWords = 8;  // column words (256 terms, one 32-byte sector per column) per warp and turn
constexpr int kClosePitch = 9;  // padded row of the anticommutation words (bank conflicts)

// Word j of a gate's columns after the first four, and of the parity column for odd generators.
__device__ __forceinline__ uint32_t more_columns(const GateDesc &gd, const Store &st, uint32_t parity_col, uint32_t j) {
    uint32_t a = 0;
    if (gd.n_fold <= kMaxFoldCols) {
        for (int f = 4; f < gd.n_fold; ++f) a ^= st.cols[static_cast<uint64_t>(gd.fold_cols[f]) * st.cstride + j];
    }
    else {
        for (uint32_t wd = 0; wd < parity_col / 64; ++wd)
            for (uint64_t x = gd.fold[wd]; x != 0; x &= x - 1)
                a ^= st.cols[(64ull * wd + __ffsll(static_cast<long long>(x)) - 1) * st.cstride + j];
    }
    if (gd.g_odd != 0) a ^= st.cols[static_cast<uint64_t>(parity_col) * st.cstride + j];
    return a;
}

// Applies the pending window (ctl) to its passive terms and collects the candidates of the next window, of at most
// kWindow gates from cnt->step on and before hi. Bound by memory: 16 bytes of coefficient per term and the columns of
// the window's gates, against 64 bytes per anticommuting (term, gate) pair when done gate by gate. A warp takes 8
// column words: eight lanes form one gate's words (one 32-byte sector per column), the words go through shared memory
// to a bit transposition, and every lane then holds the gate mask of its own term.
__global__ void __launch_bounds__(kCloseWarps * 32, 4)
    k_window_close(Store st, uint32_t parity_col, WindowScratch ws, uint32_t *__restrict__ cand, const Counters *__restrict__ cnt,
                   const GateDesc *__restrict__ gates, uint32_t L, uint32_t hi, Trunc tr, uint64_t *__restrict__ stats) {
    __shared__ __align__(16) uint32_t s_word[kCloseWarps][kWindow * kClosePitch];
    static_assert(sizeof(TableWork) <= sizeof(s_word), "the tables are built in the transposition buffers");
    __shared__ double s_cos[kWindow];
    __shared__ __align__(16) const uint32_t *s_col[kWindow][4]; // first fold columns, nullptr past the last
    __shared__ uint8_t s_more[kWindow]; // 1: the gate has further columns (or the parity column)
    __shared__ uint32_t s_anti[kWindow];
    __shared__ double s_smax[kWindow];
    WindowCtl *ctl = ws.ctl;
    const uint32_t done = ctl->pending ? ctl->gates : 0u;
    const uint32_t lo = ctl->lo;
    const uint64_t n_start = done ? ctl->n_start : 0;
    const uint64_t n_now = cnt->n;
    const uint32_t next_lo = cnt->step;
    const uint32_t next_hi = next_lo + window_length(kLengths - 1, hi > next_lo ? hi - next_lo : 0u);
    const bool next = next_hi > next_lo && cnt->stall == kNoStall;
    if (next)
        for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < kLengths * kMaxSectors; k += gridDim.x * blockDim.x) {
            ctl->load[0][k] = 0;
            if (k < kMaxSectors) {
                ctl->sector[k] = 0;
                ctl->filled[k] = 0;
            }
        }
    if (blockIdx.x == 0 && threadIdx.x < done) {
        // the per-gate counters: store size, emitted branches, and the appends' share of the anticommuting
        // terms (the terms below n_start are counted from the columns below)
        uint64_t n = n_start;
        for (uint32_t g = 0; g < threadIdx.x; ++g) n += ctl->appended[g];
        uint64_t *s = stats + 4 * static_cast<uint64_t>(lo + threadIdx.x);
        s[0] = n;
        s[2] = ctl->emitted[threadIdx.x];
        if (ctl->anti[threadIdx.x] != 0)
            atomicAdd(reinterpret_cast<unsigned long long *>(s) + 1, static_cast<unsigned long long>(ctl->anti[threadIdx.x]));
    }
    if (done == 0 && !next) return;
    if (blockIdx.x == gridDim.x - 1) { // the last block prepares the next window's tables while the others stream
        if (next)
            window_tables(gates, L, next_lo, static_cast<int>(next_hi - next_lo), static_cast<int>(parity_col / 64),
                          ctl->tables, ctl->comm, *reinterpret_cast<TableWork *>(&s_word[0][0]));
        return;
    }
    const uint32_t blocks = gridDim.x - 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < kWindow) {
        const int g = static_cast<int>(threadIdx.x);
        s_anti[g] = 0;
        if (g < static_cast<int>(done)) {
            const GateDesc &gd = gates[L - 1 - (lo + g)];
            s_cos[g] = gd.cosv;
            const int nf = gd.empty || gd.n_fold > kMaxFoldCols ? 0 : gd.n_fold;
            s_more[g] = gd.n_fold > 4 || gd.g_odd != 0;
#pragma unroll
            for (int f = 0; f < 4; ++f)
                s_col[g][f] = f < nf ? st.cols + static_cast<uint64_t>(gd.fold_cols[f]) * st.cstride : nullptr;
        }
        s_smax[g] = next && next_lo + g < next_hi ? gates[L - 1 - (next_lo + g)].abs_sin : 0.0;
    }
    __syncthreads();
    double smax = 0.0;
    if (next)
        for (uint32_t g = 0; g < next_hi - next_lo; ++g) smax = max_or_nan(smax, s_smax[g]);
    uint32_t *sw = s_word[warp];
    const uint32_t nw_start = static_cast<uint32_t>((n_start + 31) >> 5);
    const uint32_t tail = (n_start & 31) ? ((1u << (n_start & 31)) - 1u) : 0xFFFFFFFFu;
    const uint32_t n_units = static_cast<uint32_t>((n_now + 32 * kCloseWords - 1) / (32 * kCloseWords));
    uint32_t cnt0 = 0, cnt1 = 0; // anticommuting terms of gates `lane` and `lane + 32`
    for (uint32_t u = blockIdx.x * kCloseWarps + warp; u < n_units; u += blocks * kCloseWarps) {
        const uint32_t j0 = u * kCloseWords;
        double c[kCloseWords];
#pragma unroll
        for (int w = 0; w < kCloseWords; ++w) {
            const uint64_t i = static_cast<uint64_t>(j0 + w) * 32 + lane;
            c[w] = i < n_now ? st.coef[i] : 0.0;
        }
        const bool flush = j0 < nw_start; // warp-uniform
        uint32_t actw = 0;
        if (flush) {
            if (lane < kCloseWords && j0 + lane < nw_start) actw = ws.act[j0 + lane];
            const int w = lane & 7;
            const uint32_t j = j0 + w;
            for (int g0 = 0; g0 < static_cast<int>(done); g0 += 16) {
                // four gates per lane and turn, up to 16 column loads in flight (two gates: 4 % longer)
                uint32_t anti[4] = {0, 0, 0, 0};
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const int g = g0 + 4 * h + (lane >> 3);
                    if (g < static_cast<int>(done) && j < nw_start) {
                        uint32_t v[4];
#pragma unroll
                        for (int f = 0; f < 4; ++f) {
                            const uint32_t *col = s_col[g][f];
                            v[f] = col != nullptr ? col[j] : 0u;
                        }
                        anti[h] = v[0] ^ v[1] ^ v[2] ^ v[3];
                        if (s_more[g]) {
                            anti[h] ^= more_columns(gates[L - 1 - (lo + g)], st, parity_col, j);
                        }
                        if (j == nw_start - 1) anti[h] &= tail;
                    }
                }
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const int g = g0 + 4 * h + (lane >> 3);
                    if (g < kWindow) sw[g * kClosePitch + w] = anti[h];
                }
            }
            __syncwarp();
        }
        uint32_t cb[kCloseWords];
        uint32_t n_cb = 0;
#pragma unroll
        for (int w = 0; w < kCloseWords; ++w) {
            const uint64_t i = static_cast<uint64_t>(j0 + w) * 32 + lane;
            if (flush) {
                const uint32_t a0 = lane < static_cast<int>(done) ? sw[lane * kClosePitch + w] : 0u;
                cnt0 += __popc(a0);
                uint32_t m0 = transpose32(a0, lane), m1 = 0;
                if (done > 32) {
                    const uint32_t a1 = lane + 32 < static_cast<int>(done) ? sw[(lane + 32) * kClosePitch + w] : 0u;
                    cnt1 += __popc(a1);
                    m1 = transpose32(a1, lane);
                }
                const uint32_t active = __shfl_sync(0xFFFFFFFFu, actw, w);
                if (((active >> lane) & 1u) == 0 && (m0 | m1) != 0) {
                    double x = c[w];
                    for (; m0 != 0; m0 &= m0 - 1) x *= s_cos[__ffs(static_cast<int>(m0)) - 1];
                    for (; m1 != 0; m1 &= m1 - 1) x *= s_cos[__ffs(static_cast<int>(m1)) + 31];
                    c[w] = x;
                    st.coef[i] = x;
                }
            }
            const bool may = next && i < n_now && !(tr.has_lower && smax * fabs(c[w]) <= tr.lower);
            cb[w] = __ballot_sync(0xFFFFFFFFu, may);
            n_cb += __popc(cb[w]);
        }
        __syncwarp();
        if (next) {
            if (lane < kCloseWords) ws.act[j0 + lane] = 0u;
            if (n_cb != 0) {
                uint32_t base = 0;
                if (lane == 0) base = atomicAdd(&ctl->n_cand, n_cb);
                base = __shfl_sync(0xFFFFFFFFu, base, 0);
#pragma unroll
                for (int w = 0; w < kCloseWords; ++w) {
                    if ((cb[w] >> lane) & 1u) cand[base + __popc(cb[w] & ((1u << lane) - 1u))] = (j0 + w) * 32 + lane;
                    base += __popc(cb[w]);
                }
            }
        }
    }
    if (done != 0) {
        if (cnt0) atomicAdd(&s_anti[lane], cnt0);
        if (cnt1) atomicAdd(&s_anti[lane + 32], cnt1);
        __syncthreads();
        if (threadIdx.x < done && s_anti[threadIdx.x] != 0)
            atomicAdd(reinterpret_cast<unsigned long long *>(stats + 4 * static_cast<uint64_t>(lo + threadIdx.x)) + 1,
                      static_cast<unsigned long long>(s_anti[threadIdx.x]));
    }
}

// ----- the sectors' lists ---------------------------------------------------------------------------------------

// Gates (bit j) whose generator anticommutes with key m, and its f for the window lengths [I, I + N): XOR of the
// rows of m's set bits.
template <int W, int N>
__device__ __forceinline__ uint64_t window_mask(const uint64_t (&m)[W], const uint64_t *mask_rows, const uint32_t *inv_rows,
                                                uint64_t odd, uint32_t (&f)[N]) {
    uint64_t mask = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) f[i] = 0;
    int pop = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        pop += __popcll(m[w]);
        for (uint64_t x = m[w]; x != 0; x &= x - 1) {
            const int c = 64 * w + __ffsll(static_cast<long long>(x)) - 1;
            mask ^= mask_rows[c];
#pragma unroll
            for (int i = 0; i < N; ++i) f[i] ^= inv_rows[i * 64 * W + c];
        }
    }
    return (pop & 1) ? mask ^ odd : mask;
}

// Whether a term of |coefficient| av may pass the lower_atol gate of some gate in `mask` (sin: |sin| of the
// gates). In floats, each rounded so that no term that passes is lost; NaN passes.
__device__ __forceinline__ bool may_emit(uint64_t mask, double av, const float *sin, const Trunc &tr) {
    if (mask == 0) return false;
    if (!tr.has_lower) return true;
    float smax = 0.0f;
    for (uint64_t x = mask; x != 0; x &= x - 1) {
        const float s = sin[__ffsll(static_cast<long long>(x)) - 1];
        smax = (s > smax || s != s) ? s : smax;
    }
    return !(__fmul_ru(smax, __double2float_ru(av)) <= __double2float_rd(tr.lower));
}

// Too many candidates for a window to pay (kDenseTerms, kLargeTerms).
__device__ __forceinline__ bool window_dense(uint64_t n_cand, uint64_t n) {
    return n > kDenseTerms && n_cand > (n > kLargeTerms ? n / 4 : n / 2);
}

__device__ __forceinline__ uint64_t first_gates(uint32_t n) { return n >= 64 ? ~0ull : (1ull << n) - 1ull; }

// The sectors' loads (anticommuting gates of their active terms) for every window length, from a sample of the
// candidates: enough to tell a balanced length from one with a few large cosets.
constexpr uint32_t kSampleBlocks = 64, kSamplePerThread = 2;
template <int W>
__global__ void __launch_bounds__(256) k_window_sample(Store st, WindowScratch ws, const uint32_t *__restrict__ cand,
                                                        const Counters *__restrict__ cnt, uint32_t hi, uint32_t sectors,
                                                        Trunc tr) {
    __shared__ uint64_t s_mask[64 * W];
    __shared__ uint32_t s_inv[kLengths][64 * W];
    __shared__ uint32_t s_load[kLengths][kMaxSectors];
    __shared__ float s_sin[kWindow];
    WindowCtl *ctl = ws.ctl;
    const uint32_t lo = cnt->step;
    if (cnt->stall != kNoStall || lo >= hi) return;
    const uint32_t n = ctl->n_cand, most = hi - lo;
    if (n <= blockIdx.x * blockDim.x || window_dense(n, cnt->n)) return;
    for (uint32_t c = threadIdx.x; c < 64 * W; c += blockDim.x) {
        s_mask[c] = ctl->tables.mask[c];
#pragma unroll
        for (int i = 0; i < kLengths; ++i) s_inv[i][c] = ctl->tables.inv[i][c];
    }
    if (threadIdx.x < kWindow) s_sin[threadIdx.x] = __double2float_ru(ctl->tables.sin[threadIdx.x]);
    for (uint32_t k = threadIdx.x; k < kLengths * kMaxSectors; k += blockDim.x) s_load[0][k] = 0;
    __syncthreads();
    // sample k of all is candidate k * n / samples (every candidate when there are fewer)
    const uint32_t all = gridDim.x * blockDim.x * kSamplePerThread, samples = min(n, all);
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < samples; k += gridDim.x * blockDim.x) {
        const uint32_t idx = cand[static_cast<uint64_t>(k) * n / samples];
        const double av = fabs(st.coef[idx]);
        uint64_t m[W];
        load_key<W>(st.keys, idx, m);
        uint32_t f[kLengths];
        const uint64_t mask = window_mask<W, kLengths>(m, s_mask, s_inv[0], ctl->tables.odd, f);
#pragma unroll
        for (int i = 0; i < kLengths; ++i) {
            const uint64_t in = mask & first_gates(window_length(i, most));
            if (may_emit(in, av, s_sin, tr)) atomicAdd(&s_load[i][mix64(f[i]) % sectors], static_cast<uint32_t>(__popcll(in)));
        }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < kLengths * kMaxSectors; k += blockDim.x)
        if (s_load[0][k] != 0) atomicAdd(&ctl->load[0][k], s_load[0][k]);
}

// The window length to run, by the whole block, or -1 when the gates take less time one by one (all in picoseconds).
//   Windows, per gate: a sector's block takes about 2.5 us plus 0.05 us for each anticommuting term of the busiest sector
//   (from the 33rd on, against gate by gate: the length that spreads the terms best is the better one anyhow); a window's
//   other launches 150 us plus 20 ps per term of the store (the dense pass), spread over its gates.
//   Gate by gate: 6.2 us for the two launches, up to 4 us for the chain of the branches, 65 ps per anticommuting
//   active term and 1.5 ps per term (measured from 1 to 3e6 terms: 5.6 us at a few terms, 12 at 3e5 with 2e4 active and
//   anticommuting, 33 at 1e6 with 4e5).
// Up to 1.15 times that, windows go on (a declined try and the way back cost as much), and 0.2 ms over the gates that
// are left in favour of windows: what a change over costs. Measured on lines and lattices, windows against gate by
// gate: 2.0 times as long over 8 gates, 1.2 over 32, 0.8 over 64; on 8 to 11 qubits without truncation, where no
// length but the shortest is balanced, 1.2 to 2.2. In whole numbers: every block of the two kernels that ask (count,
// which makes the masks, and scatter, which sets the window up) has to come to the same length, and floating-point
// sums may be contracted differently in each.
struct LengthShared {
    uint32_t most[kLengths], sum[kLengths];
};
__device__ __forceinline__ int choose_length(const WindowCtl *ctl, uint32_t sectors, uint32_t most, uint64_t n, LengthShared &s) {
    if (threadIdx.x < kLengths) s.most[threadIdx.x] = s.sum[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kLengths; ++i) {
        uint32_t m = 0, t = 0;
        for (uint32_t k = threadIdx.x; k < sectors; k += blockDim.x) {
            m = max(m, ctl->load[i][k]);
            t += ctl->load[i][k];
        }
        m = __reduce_max_sync(0xFFFFFFFFu, m);
        t = __reduce_add_sync(0xFFFFFFFFu, t);
        if ((threadIdx.x & 31) == 0) {
            atomicMax(&s.most[i], m);
            atomicAdd(&s.sum[i], t);
        }
    }
    __syncthreads();
    constexpr uint64_t all = kSampleBlocks * 256 * kSamplePerThread; // 2^15 samples of at most 2^6 gates each
    const uint64_t n_cand = ctl->n_cand;
    auto scaled = [&](uint32_t load) { return n_cand > all ? load * n_cand / all : load; }; // the product is below 2^53
    int best = kLengths - 1;
    uint64_t t_best = 0;
    for (int i = kLengths - 1; i >= 0; --i) {
        const uint64_t t = 2500000 + (50000 * scaled(s.most[i]) + 150000000 + 20 * n) / window_length(i, most);
        if (i == kLengths - 1 || t < t_best) {
            best = i;
            t_best = t;
        }
    }
    const uint64_t len = window_length(best, most), active = scaled(s.sum[best]) / len;
    t_best -= 50000 * min(scaled(s.most[best]) / len, uint64_t(32));
    const uint64_t by_gate = 6200000 + 4000 * min(active, uint64_t(1000)) + 65 * active + 3 * n / 2;
    const uint64_t change = 200000000 / window_length(kLengths - 1, most);
    return 20 * t_best <= 23 * by_gate + 20 * change ? best : -1;
}

// Mask and sector of every candidate; one that passes no lower_atol gate of a gate of the window it
// anticommutes with gets no sector. Bound by the candidates' key rows (scattered, 8W + 8 bytes).
template <int W>
__global__ void __launch_bounds__(256) k_window_count(Store st, WindowScratch ws, const uint32_t *__restrict__ cand,
                                                       uint64_t *__restrict__ c_mask, uint16_t *__restrict__ c_sector,
                                                       const Counters *__restrict__ cnt, uint32_t hi, uint32_t sectors,
                                                       Trunc tr) {
    __shared__ uint64_t s_mask[64 * W];
    __shared__ uint32_t s_inv[64 * W];
    __shared__ uint32_t s_entries[kMaxSectors];
    __shared__ float s_sin[kWindow];
    __shared__ LengthShared s_len;
    WindowCtl *ctl = ws.ctl;
    const uint32_t lo = cnt->step;
    if (cnt->stall != kNoStall || lo >= hi) return;
    const uint32_t n = ctl->n_cand;
    if (n <= blockIdx.x * blockDim.x || window_dense(n, cnt->n)) return;
    const int len = choose_length(ctl, sectors, hi - lo, cnt->n, s_len);
    if (len < 0) return;
    const uint64_t in = first_gates(window_length(len, hi - lo));
    for (uint32_t c = threadIdx.x; c < 64 * W; c += blockDim.x) {
        s_mask[c] = ctl->tables.mask[c];
        s_inv[c] = ctl->tables.inv[len][c];
    }
    if (threadIdx.x < kWindow) s_sin[threadIdx.x] = __double2float_ru(ctl->tables.sin[threadIdx.x]);
    for (uint32_t k = threadIdx.x; k < kMaxSectors; k += blockDim.x) s_entries[k] = 0;
    __syncthreads();
    const uint64_t odd = ctl->tables.odd;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t idx = cand[k];
        const double av = fabs(st.coef[idx]);
        uint64_t m[W];
        load_key<W>(st.keys, idx, m);
        uint32_t f[1];
        const uint64_t mask = window_mask<W, 1>(m, s_mask, s_inv, odd, f) & in;
        uint16_t sector = kNoSector;
        if (may_emit(mask, av, s_sin, tr)) {
            sector = static_cast<uint16_t>(mix64(f[0]) % sectors);
            atomicAdd(&s_entries[sector], 1u);
        }
        c_sector[k] = sector;
        c_mask[k] = mask;
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < sectors; k += blockDim.x)
        if (s_entries[k] != 0) atomicAdd(&ctl->sector[k], s_entries[k]);
}

// First chunk of every sector (exclusive prefix of the chunk counts) into s_base[0 .. sectors], by the block.
__device__ __forceinline__ void sector_bases(const uint32_t *entries, uint32_t sectors, uint32_t *s_base, uint32_t *s_part) {
    const uint32_t per = (sectors + blockDim.x - 1) / blockDim.x;
    uint32_t sum = 0;
    for (uint32_t i = 0; i < per; ++i) {
        const uint32_t k = threadIdx.x * per + i;
        if (k < sectors) sum += (entries[k] + kChunk - 1) / kChunk;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += x;
    }
    if (lane == 31) s_part[warp] = incl;
    __syncthreads();
    uint32_t acc = incl - sum;
    for (int w = 0; w < warp; ++w) acc += s_part[w];
    for (uint32_t i = 0; i < per; ++i) {
        const uint32_t k = threadIdx.x * per + i;
        if (k < sectors) {
            s_base[k] = acc;
            acc += (entries[k] + kChunk - 1) / kChunk;
            if (k + 1 == sectors) s_base[sectors] = acc;
        }
    }
    __syncthreads();
}

// Places the candidates on their sectors' lists. A block takes a contiguous share of the candidates and
// reserves its places sector by sector (one counter bump per sector it holds).
__global__ void __launch_bounds__(256) k_window_scatter(Store st, WindowScratch ws, const uint32_t *__restrict__ cand,
                                                         const uint64_t *__restrict__ c_mask,
                                                         const uint16_t *__restrict__ c_sector,
                                                         const Counters *__restrict__ cnt, uint32_t hi, uint32_t sectors) {
    __shared__ uint32_t s_base[kMaxSectors + 1], s_at[kMaxSectors], s_part[8];
    __shared__ LengthShared s_len;
    WindowCtl *ctl = ws.ctl;
    const uint32_t lo = cnt->step;
    const bool run = cnt->stall == kNoStall && lo < hi;
    const uint32_t n = ctl->n_cand;
    if (run && n == 0 && blockIdx.x != 0) return;
    const int len = run && !window_dense(n, cnt->n) ? choose_length(ctl, sectors, hi - lo, cnt->n, s_len) : -1;
    if (len < 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            ctl->run = 0;
            ctl->overflow = run ? 3 : 0;
        }
        return;
    }
    const uint32_t K = window_length(len, hi - lo);
    sector_bases(ctl->sector, sectors, s_base, s_part);
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) {
            ctl->run = 1;
            ctl->lo = lo;
            ctl->gates = K;
            ctl->overflow = 0;
            ctl->n_start = cnt->n;
            ctl->n_chunks = s_base[sectors];
            ctl->grow = max(kGrowChunks, 8 * (n / sectors) / kChunk);
        }
        if (threadIdx.x < kWindow) {
            ctl->anti[threadIdx.x] = 0;
            ctl->emitted[threadIdx.x] = 0;
            ctl->appended[threadIdx.x] = 0;
        }
    }
    const uint32_t share = (n + gridDim.x - 1) / gridDim.x;
    const uint32_t c_lo = min(n, share * blockIdx.x), c_hi = min(n, c_lo + share);
    if (c_lo == c_hi) return;
    for (uint32_t k = threadIdx.x; k < sectors; k += blockDim.x) s_at[k] = 0;
    __syncthreads();
    for (uint32_t k = c_lo + threadIdx.x; k < c_hi; k += blockDim.x) {
        const uint16_t s = c_sector[k];
        if (s != kNoSector) atomicAdd(&s_at[s], 1u);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < sectors; k += blockDim.x) {
        const uint32_t c = s_at[k];
        s_at[k] = c != 0 ? s_base[k] * kChunk + atomicAdd(&ctl->filled[k], c) : 0u;
    }
    __syncthreads();
    for (uint32_t k0 = c_lo + threadIdx.x; k0 < c_hi; k0 += 4 * blockDim.x) { // four candidates in flight per thread
        uint16_t s[4];
        uint32_t idx[4];
        uint64_t mask[4];
        double v[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint32_t k = k0 + r * blockDim.x;
            s[r] = k < c_hi ? c_sector[k] : kNoSector;
            idx[r] = k < c_hi ? cand[k] : 0u;
            mask[r] = k < c_hi ? c_mask[k] : 0ull;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) v[r] = s[r] != kNoSector ? st.coef[idx[r]] : 0.0;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            if (s[r] == kNoSector) continue;
            const uint32_t slot = atomicAdd(&s_at[s[r]], 1u);
            if (slot >= ws.slots) continue; // cannot happen: the slots hold every term of the store
            ws.a_idx[slot] = idx[r];
            ws.a_mask[slot] = mask[r];
            ws.a_val[slot] = v[r];
            ws.slot_of[idx[r]] = slot;
            atomicOr(&ws.act[idx[r] >> 5], 1u << (idx[r] & 31));
        }
    }
}

// ----- the gates of one window --------------------------------------------------------------------------------

template <int W>
struct GateW { // what the gates kernel needs of a GateDesc
    uint64_t g[W], wmask[W];
    double cosv, sinv, abs_sin, inv_cos;
    uint64_t pivot_bit;
    int32_t gpop, gy, pivot_word, pad;
};

template <int W>
struct GateShared {
    GateW<W> gd[kWindow];
    uint64_t comm[kWindow];
    uint32_t chunk[kSectorChunks]; // the sector's chunks, in list order
    uint32_t anti[kWindow], emitted[kWindow], appended[kWindow];
    uint32_t n_list[2], n_pass, n_queue, n_join, n_insert, first, most_chunks;
    int failed;
};
struct GateLists { // sized by the block's T threads
    double *pass_v, *q_v;             // [2T], [T]
    uint32_t *pass_slot, *pass_idx;   // [2T] anticommuting terms that passed the lower_atol gate
    uint32_t *q_slot, *q_tgt;         // [T] the queue; further entries go to global memory
    unsigned long long *ins_entry;    // [T] table entries of the appended terms
    uint64_t *ins_pos;                // [T] where their probes start
    uint16_t *list;                   // [16T] set bits of the turn's T / 2 slot words
    uint8_t *q_flag;                  // [T]
};
__host__ __device__ inline size_t gate_lists_bytes(uint32_t T) {
    return static_cast<size_t>(T) * (2 * 8 + 8 + 8 + 8 + 2 * 4 + 2 * 4 + 2 * 4 + 32 + 1);
}
__device__ __forceinline__ GateLists gate_lists(uint8_t *p, uint32_t T) {
    GateLists l;
    l.pass_v = reinterpret_cast<double *>(p);
    l.q_v = l.pass_v + 2 * T;
    l.ins_entry = reinterpret_cast<unsigned long long *>(l.q_v + T);
    l.ins_pos = reinterpret_cast<uint64_t *>(l.ins_entry + T);
    l.pass_slot = reinterpret_cast<uint32_t *>(l.ins_pos + T);
    l.pass_idx = l.pass_slot + 2 * T;
    l.q_slot = l.pass_idx + 2 * T;
    l.q_tgt = l.q_slot + T;
    l.list = reinterpret_cast<uint16_t *>(l.q_tgt + T);
    l.q_flag = reinterpret_cast<uint8_t *>(l.list + 16 * T);
    return l;
}
// Takes the first free table slot from pos on (the probe limit cannot be reached below load 1/2).
__device__ __forceinline__ void table_insert(const Store &st, unsigned long long entry, uint64_t pos, Counters *cnt) {
    for (uint64_t probes = 0;; ++probes) {
        if (probes > st.tmask) {
            atomicOr(&cnt->err, 2u);
            return;
        }
        if (atomicCAS(&st.table[pos], kEmptySlot, entry) == kEmptySlot) return;
        pos = (pos + 1) & st.tmask;
    }
}
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// All gates of a window on one sector per block; blocks do not wait for one another. Bound by latency: per gate
// a chain of dependent loads (slot bits, value, term, key row, table slot, candidate row, partner's value) for
// the sector's few hundred anticommuting active terms; the resident blocks of an SM overlap theirs. The lists
// are private to the block (plain cached accesses); key rows and table slots, which other blocks append to,
// are read past L1.
template <int W, int BASIS, bool MAPPED>
__global__ void __launch_bounds__(kSectorThreads, kSectorsPerSM)
    k_window_gates(Store st, Scratch sc, WindowScratch ws, Counters *cnt, const GateDesc *__restrict__ gates, uint32_t L,
                   Trunc tr) {
    extern __shared__ __align__(16) uint8_t smem[];
    GateShared<W> &sh = *reinterpret_cast<GateShared<W> *>(smem);
    const uint32_t T = blockDim.x, tid = threadIdx.x;
    const GateLists ls = gate_lists(smem + sizeof(GateShared<W>), T);
    WindowCtl *ctl = ws.ctl;
    if (ctl->run == 0) return;
    uint32_t n_ent = ctl->sector[blockIdx.x];
    if (n_ent == 0) return; // no active term, and none can join: a partner shares its source's sector
    const int lane = tid & 31;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const int K = static_cast<int>(ctl->gates);
    const uint32_t lo = ctl->lo;
    const uint64_t n_start = ctl->n_start;
    for (uint32_t j = tid; j < static_cast<uint32_t>(K); j += T) {
        const GateDesc &s = gates[L - 1 - (lo + j)];
        GateW<W> &d = sh.gd[j];
#pragma unroll
        for (int w = 0; w < W; ++w) {
            d.g[w] = s.g[w];
            d.wmask[w] = s.wmask[w];
        }
        d.cosv = s.cosv;
        d.sinv = s.sinv;
        d.abs_sin = s.abs_sin;
        d.inv_cos = s.inv_cos;
        d.pivot_bit = s.pivot_bit;
        d.gpop = s.gpop;
        d.gy = s.gy;
        d.pivot_word = s.pivot_word;
        sh.comm[j] = ctl->comm[j] & first_gates(static_cast<uint32_t>(K));
        sh.anti[j] = sh.emitted[j] = sh.appended[j] = 0;
    }
    if (tid == 0) {
        sh.n_list[0] = sh.n_list[1] = 0;
        sh.n_pass = sh.n_queue = sh.n_join = sh.n_insert = 0;
        sh.first = 0;
        sh.failed = 0;
    }
    __syncthreads();
    {
        uint32_t before = 0; // chunks of the sectors before this one
        for (uint32_t k = tid; k < blockIdx.x; k += T) before += (ctl->sector[k] + kChunk - 1) / kChunk;
        before = __reduce_add_sync(0xFFFFFFFFu, before);
        if (lane == 0 && before != 0) atomicAdd(&sh.first, before);
    }
    __syncthreads();
    const uint32_t first = sh.first;
    uint32_t n_chunks = (n_ent + kChunk - 1) / kChunk;
    if (n_chunks > kSectorChunks) {
        if (tid == 0) ctl->overflow = 2;
        return;
    }
    if (tid == 0) sh.most_chunks = min(kSectorChunks, max(ctl->grow, 4 * n_chunks)); // read by the same thread
    for (uint32_t k = tid; k < n_chunks; k += T) sh.chunk[k] = first + k;
    __syncthreads();
    auto slot_at = [&](uint32_t p) { return sh.chunk[p / kChunk] * kChunk + p % kChunk; };
    // slot bits of the entries from the start
    for (uint32_t w = tid >> 5; w < (n_ent + 31) / 32; w += T >> 5) {
        const uint32_t p = w * 32 + lane;
        const uint64_t mask = p < n_ent ? ws.a_mask[slot_at(p)] : 0ull;
        ws.a_lead[slot_at(p)] = 0;
        uint32_t *row = ws.a_bits + static_cast<uint64_t>(sh.chunk[w / 32]) * kWindow * 32 + w % 32;
        row[lane * 32] = transpose32(static_cast<uint32_t>(mask), lane);
        row[(lane + 32) * 32] = transpose32(static_cast<uint32_t>(mask >> 32), lane);
    }
    __syncthreads();

    for (int b = 0; b < K; ++b) {
        const GateW<W> &gd = sh.gd[b];
        const double cosv = gd.cosv, sinabs = gd.abs_sin, sinv = gd.sinv;
        const uint32_t n_words = (n_ent + 31) / 32;
        uint32_t par = 0, room = n_ent; // list places this gate may need so far
        for (uint32_t w0 = 0; w0 < n_words; w0 += T / 2, par ^= 1u) {
            // the set bits of the turn's words, as (word in turn, bit)
            if (tid < T / 2) {
                const uint32_t w = w0 + tid;
                const uint32_t bits =
                    w < n_words ? ws.a_bits[(static_cast<uint64_t>(sh.chunk[w / 32]) * kWindow + b) * 32 + w % 32] : 0u;
                const int c = __popc(bits);
                int incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                    if (lane >= o) incl += x;
                }
                uint32_t at = 0;
                if (lane == 31 && incl != 0) at = atomicAdd(&sh.n_list[par], static_cast<uint32_t>(incl));
                at = __shfl_sync(0xFFFFFFFFu, at, 31) + static_cast<uint32_t>(incl - c);
                for (uint32_t x = bits; x != 0; x &= x - 1)
                    ls.list[at++] = static_cast<uint16_t>((tid << 5) | static_cast<uint32_t>(__ffs(static_cast<int>(x)) - 1));
            }
            __syncthreads();
            const uint32_t A = sh.n_list[par];
            room += A; // each of them makes at most one term join
            if (room > n_chunks * kChunk) { // block-uniform
                const uint32_t need = (room + kChunk - 1) / kChunk;
                if (tid == 0) {
                    for (uint32_t k = n_chunks; k < need; ++k) {
                        const uint32_t c = k < sh.most_chunks ? atomicAdd(&ctl->n_chunks, 1u) : 0u;
                        if (k >= sh.most_chunks || c >= ws.slots / kChunk) {
                            sh.failed = 2; // lists, not the store: its capacity may well do
                            break;
                        }
                        sh.chunk[k] = c;
                    }
                }
                __syncthreads();
                if (sh.failed != 0) { // nothing of this window is committed: its gates run one by one
                    if (tid == 0) ctl->overflow = static_cast<uint32_t>(sh.failed);
                    return;
                }
                n_chunks = need;
            }
            // In rounds of two terms per thread: values and the lower_atol gate first, then, gathered so that
            // every lane has one, the terms that passed it.
            for (uint32_t k0 = 0; k0 < A; k0 += 2 * T) {
                uint32_t slot[2], idx[2];
                double v[2];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const uint32_t k = k0 + r * T + tid;
                    slot[r] = kNoStall;
                    v[r] = 0.0;
                    idx[r] = 0;
                    if (k < A) {
                        const uint32_t e = ls.list[k];
                        slot[r] = slot_at((w0 + (e >> 5)) * 32 + (e & 31));
                        v[r] = ws.a_val[slot[r]];
                        idx[r] = ws.a_idx[slot[r]];
                    }
                }
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const bool pass = slot[r] != kNoStall && !(tr.has_lower && sinabs * fabs(v[r]) <= tr.lower);
                    if (slot[r] != kNoStall) ws.a_val[slot[r]] = v[r] * cosv;
                    const uint32_t pb = __ballot_sync(0xFFFFFFFFu, pass);
                    uint32_t at = 0;
                    if (lane == 0 && pb != 0) at = atomicAdd(&sh.n_pass, static_cast<uint32_t>(__popc(pb)));
                    at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(pb & lt_mask);
                    if (pass) {
                        prefetch_l2(st.keys + static_cast<uint64_t>(idx[r]) * W);
                        ls.pass_slot[at] = slot[r];
                        ls.pass_idx[at] = idx[r];
                        ls.pass_v[at] = v[r];
                    }
                }
                __syncthreads();
                const uint32_t P = sh.n_pass;
                for (uint32_t k1 = 0; k1 < P; k1 += T) {
                    const uint32_t k = k1 + tid;
                    bool hit = false, miss = false, follower = false;
                    int phase = 0;
                    uint32_t s_slot = 0, found = 0;
                    uint64_t p[W], pos = 0, mask = 0;
                    double vs = 0.0;
                    uint32_t tag = 0;
                    if (k < P) {
                        s_slot = ls.pass_slot[k];
                        vs = ls.pass_v[k];
                        uint64_t m[W];
                        load_key_l2<W>(st.keys, ls.pass_idx[k], m);
                        int mpop = 0, ov = 0;
#pragma unroll
                        for (int w = 0; w < W; ++w) {
                            p[w] = m[w] ^ gd.g[w];
                            mpop += __popcll(m[w]);
                            ov += __popcll(m[w] & gd.g[w]);
                        }
                        const int ppop = mpop + gd.gpop - 2 * ov;
                        bool keep;
                        if constexpr (MAPPED) keep = keep_partner_mapped<W>(p, tr);
                        else keep = keep_partner<W>(p, ppop, tr);
                        if (keep || (tr.has_upper && sinabs * fabs(vs) >= tr.upper)) {
                            const uint64_t h = key_hash<W>(p);
                            pos = h & st.tmask;
                            unsigned long long ts = __ldcg(st.table + pos);
                            mask = ws.a_mask[s_slot] ^ sh.comm[b]; // the partner's
#pragma unroll
                            for (int w = 0; w < W; ++w)
                                if (w == gd.pivot_word) follower = (m[w] & gd.pivot_bit) != 0;
                            if (!follower) ws.a_lead[s_slot] = static_cast<uint8_t>(b + 1);
                            phase = rotation_phase<W, BASIS>(m, p, gd, mpop, ppop);
                            tag = static_cast<uint32_t>(h >> 32);
                            miss = true;
                            for (uint64_t probes = 0; ts != kEmptySlot; ++probes) {
                                if (probes > st.tmask) { // a full table cannot happen below load 1/2; never spin
                                    atomicOr(&cnt->err, 1u);
                                    miss = false;
                                    break;
                                }
                                if (static_cast<uint32_t>(ts >> 32) == tag) {
                                    found = static_cast<uint32_t>(ts);
                                    uint64_t o[W];
                                    load_key_l2<W>(st.keys, found, o);
                                    prefetch_l2(ws.slot_of + found);
                                    bool eq = true;
#pragma unroll
                                    for (int w = 0; w < W; ++w) eq = eq && o[w] == p[w];
                                    if (eq) {
                                        hit = true;
                                        miss = false;
                                        break;
                                    }
                                }
                                pos = (pos + 1) & st.tmask;
                                ts = __ldcg(st.table + pos);
                            }
                        }
                    }
                    const uint32_t hb = __ballot_sync(0xFFFFFFFFu, hit);
                    uint32_t qb = 0;
                    if (lane == 0 && hb != 0) qb = atomicAdd(&sh.n_queue, static_cast<uint32_t>(__popc(hb)));
                    qb = __shfl_sync(0xFFFFFFFFu, qb, 0) + __popc(hb & lt_mask);
                    if (hit) {
                        const uint8_t flag = static_cast<uint8_t>((follower ? 1 : 0) | (phase_code(phase) << 1));
                        if (qb < T) {
                            ls.q_flag[qb] = flag;
                            ls.q_v[qb] = vs;
                            ls.q_slot[qb] = s_slot;
                            ls.q_tgt[qb] = found;
                        }
                        else { // at most one branch per list entry: the sector's own slots hold the rest of the queue
                            const uint32_t q = slot_at(qb);
                            sc.q_src[q] = s_slot;
                            sc.q_flag[q] = flag;
                            sc.q_val[q] = vs;
                            ws.q_tgt[q] = found;
                        }
                    }
                    // A missing partner is appended at once: only this term's gate-b branch leads to it, and the
                    // gate does not touch it further.
                    const uint32_t mb = __ballot_sync(0xFFFFFFFFu, miss);
                    if (mb != 0) {
                        const uint32_t n_miss = __popc(mb);
                        unsigned long long base = 0;
                        uint32_t at = 0;
                        if (lane == 0) {
                            base = atomicAdd(&cnt->n, static_cast<unsigned long long>(n_miss));
                            at = atomicAdd(&sh.n_join, n_miss);
                            atomicAdd(&sh.appended[b], n_miss);
                            if (base + n_miss > st.cap) sh.failed = 1;
                        }
                        base = __shfl_sync(0xFFFFFFFFu, base, 0);
                        at = __shfl_sync(0xFFFFFFFFu, at, 0);
                        if (miss && base + n_miss <= st.cap) {
                            const double ph = phase_value(phase_code(phase));
                            const uint64_t nidx = base + __popc(mb & lt_mask);
                            store_key<W>(st.keys, nidx, p);
                            double c_new = (sinv * ph) * vs; // Heisenberg: the new term starts from 0
                            if (tr.schr) {
                                // Schrodinger (FusedApply.h:39-83): the new slot starts from its reference-state
                                // score and the pair rotates as a hit does
                                const double vt0 = state_score<W, BASIS>(p, tr.occ);
                                ws.a_val[s_slot] = __fma_rn(sinv * -ph, vt0, vs * cosv);
                                c_new = __fma_rn(cosv, vt0, (sinv * ph) * vs);
                            }
                            const uint32_t slot = slot_at(n_ent + at + __popc(mb & lt_mask));
                            ws.a_idx[slot] = static_cast<uint32_t>(nidx);
                            ws.a_mask[slot] = mask;
                            ws.a_val[slot] = c_new;
                            ws.a_lead[slot] = 0;
                            ws.slot_of[nidx] = slot;
                            // the appended term's share of the later gates' anticommuting counts
                            for (uint64_t x = b < 63 ? mask >> (b + 1) : 0ull; x != 0; x &= x - 1)
                                atomicAdd(&sh.anti[b + __ffsll(static_cast<long long>(x))], 1u);
                            // its table slot is taken in the resolve phase below, where nobody waits for it
                            const unsigned long long entry = (static_cast<unsigned long long>(tag) << 32) | nidx;
                            const uint32_t q = atomicAdd(&sh.n_insert, 1u);
                            if (q < T) {
                                ls.ins_entry[q] = entry;
                                ls.ins_pos[q] = pos;
                            }
                            else {
                                __threadfence();
                                table_insert(st, entry, pos, cnt);
                            }
                        }
                    }
                }
                __syncthreads();
                if (tid == 0) sh.n_pass = 0;
                __syncthreads();
            }
            if (tid == 0) sh.n_list[par] = 0;
        }
        __syncthreads();
        if (sh.failed != 0) { // the appends do not fit: nothing is committed, the host grows the store
            if (tid == 0) ctl->overflow = 1;
            return;
        }
        const uint32_t n_insert = min(sh.n_insert, T);
        if (n_insert != 0) {
            __threadfence(); // the appended rows before their table slots: other blocks may probe them
            for (uint32_t k = T - 1 - tid; k < n_insert; k += T) table_insert(st, ls.ins_entry[k], ls.ins_pos[k], cnt);
        }
        const uint32_t Q = sh.n_queue;
        for (uint32_t k = tid; k < Q; k += T) {
            uint32_t s_slot, found;
            uint8_t flag;
            double v;
            if (k < T) {
                found = ls.q_tgt[k];
                flag = ls.q_flag[k];
                v = ls.q_v[k];
                s_slot = ls.q_slot[k];
            }
            else {
                const uint32_t q = slot_at(k);
                found = ws.q_tgt[q];
                flag = sc.q_flag[q];
                v = sc.q_val[q];
                s_slot = sc.q_src[q];
            }
            const double ph = phase_value(static_cast<uint8_t>(flag >> 1));
            const uint32_t t_slot = ws.slot_of[found]; // meaningful for an active term
            const bool active = found >= n_start || ((__ldcg(ws.act + (found >> 5)) >> (found & 31)) & 1u) != 0;
            if (active) {
                const double cf = ws.a_val[t_slot]; // scaled by this gate above
                if ((flag & 1) == 0 || ws.a_lead[t_slot] != static_cast<uint8_t>(b + 1)) {
                    const double vt = cf * gd.inv_cos;
                    ws.a_val[s_slot] = __fma_rn(sinv * -ph, vt, v * cosv);
                    ws.a_val[t_slot] = __fma_rn(sinv * ph, v, cf);
                }
            }
            else {
                // still passive: its cos factors up to and including this gate's, and a place on the list
                double cf = st.coef[found];
                const uint64_t mask = ws.a_mask[s_slot] ^ sh.comm[b];
                for (uint64_t x = mask & ((1ull << b) - 1ull); x != 0; x &= x - 1)
                    cf *= sh.gd[__ffsll(static_cast<long long>(x)) - 1].cosv;
                cf *= cosv;
                const double vt = cf * gd.inv_cos;
                ws.a_val[s_slot] = __fma_rn(sinv * -ph, vt, v * cosv);
                const uint32_t slot = slot_at(n_ent + atomicAdd(&sh.n_join, 1u));
                ws.a_idx[slot] = found;
                ws.a_mask[slot] = mask;
                ws.a_val[slot] = __fma_rn(sinv * ph, v, cf);
                ws.a_lead[slot] = 0;
                ws.slot_of[found] = slot;
                atomicOr(&ws.act[found >> 5], 1u << (found & 31));
            }
        }
        __syncthreads();
        const uint32_t n_join = sh.n_join;
        // the slot bits of the terms that joined; the word they start in is written again as a whole
        if (n_join != 0)
            for (uint32_t w = n_ent / 32 + (tid >> 5); w < (n_ent + n_join + 31) / 32; w += T >> 5) {
                const uint32_t q = w * 32 + lane;
                const uint64_t m = q < n_ent + n_join ? ws.a_mask[slot_at(q)] : 0ull;
                uint32_t *row = ws.a_bits + static_cast<uint64_t>(sh.chunk[w / 32]) * kWindow * 32 + w % 32;
                row[lane * 32] = transpose32(static_cast<uint32_t>(m), lane);
                row[(lane + 32) * 32] = transpose32(static_cast<uint32_t>(m >> 32), lane);
            }
        n_ent += n_join;
        __syncthreads();
        if (tid == 0) {
            sh.emitted[b] = Q + sh.appended[b];
            sh.n_queue = 0;
            sh.n_join = 0;
            sh.n_insert = 0;
        }
    }
    __syncthreads();
    for (uint32_t k = tid; k < n_chunks; k += T) ws.fill[sh.chunk[k]] = n_ent > k * kChunk ? min(kChunk, n_ent - k * kChunk) : 0u;
    for (uint32_t j = tid; j < static_cast<uint32_t>(K); j += T) {
        if (sh.anti[j] != 0) atomicAdd(&ctl->anti[j], sh.anti[j]);
        if (sh.emitted[j] != 0) atomicAdd(&ctl->emitted[j], sh.emitted[j]);
        if (sh.appended[j] != 0) atomicAdd(&ctl->appended[j], sh.appended[j]);
    }
}

// In a captured sequence, between windows and gates that run by the per-gate kernels: goes on at step `next` if
// the windows have ended at step `at`, and stops the sequence for the host otherwise (other angles, other lengths).
__global__ void k_window_handover(Counters *cnt, uint32_t at, uint32_t next) {
    if (cnt->stall != kNoStall) return;
    if (cnt->step == at) {
        cnt->step = next;
    }
    else {
        cnt->stall = cnt->step;
        cnt->reason = kStallDense;
    }
}

// Writes the lists' values back to the store and builds the bit-columns of the window's appends (k_columns).
// A window that did not fit leaves the store as it was: the size is reset and the step recorded for the host,
// which rebuilds the table when it grows the store.
template <int W>
__global__ void __launch_bounds__(kBlock) k_window_commit(Store st, WindowScratch ws, Counters *cnt) {
    __shared__ uint32_t s_col[kBlock / 32][64][8];
    WindowCtl *ctl = ws.ctl;
    if (ctl->overflow != 0 || ctl->run == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            ctl->pending = 0;
            ctl->n_cand = 0;
            if (ctl->overflow != 0) {
                if (ctl->overflow != 3) cnt->n = ctl->n_start;
                cnt->stall = cnt->step;
                cnt->reason = ctl->overflow == 1 ? kStallStore : ctl->overflow == 2 ? kStallSector : kStallDense;
            }
        }
        return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ctl->pending = 1;
        ctl->n_cand = 0;
        cnt->step = ctl->lo + ctl->gates;
    }
    const uint32_t n_chunks = ctl->n_chunks;
    for (uint32_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
        const uint32_t n = ws.fill[c];
        uint32_t idx[kChunk / kBlock];
        double v[kChunk / kBlock];
#pragma unroll
        for (uint32_t r = 0; r < kChunk / kBlock; ++r) {
            const uint32_t k = r * kBlock + threadIdx.x;
            idx[r] = k < n ? ws.a_idx[c * kChunk + k] : kNoStall;
            v[r] = k < n ? ws.a_val[c * kChunk + k] : 0.0;
        }
#pragma unroll
        for (uint32_t r = 0; r < kChunk / kBlock; ++r)
            if (idx[r] != kNoStall) st.coef[idx[r]] = v[r];
    }
    columns_of<W>(st, ctl->n_start, cnt->n, s_col);
}

} // namespace mpx
