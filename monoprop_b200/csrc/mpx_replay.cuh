// mpx_replay.cuh -- replay of a frozen structure and its reverse sweep, in windows of gates (sm_100a).
//
// A frozen structure (MonomialPropagator.inl:620-690, Evolution.cpp:439-540) fixes which pairs every gate
// rotates; all else a gate does is to scale the other anticommuting terms by its cos. Gate by gate that is a
// scattered read and write of every anticommuting coefficient forward, a 12-byte log record each, and again a
// scattered read and write of its adjoint backward. Here a term is touched only where a gate pairs it:
//   * forward, a pair first brings its two coefficients up to date (the cos factors of the gates since the
//     last pair each was in, found from the pair's 64-bit anticommutation mask) and then rotates them; the
//     window's end brings every term up to date in one dense pass, from the bit-columns;
//   * between two pairs of a term, coefficient times adjoint is constant: kappa = c lambda. A gate j of that
//     stretch adds lambda' (-2 s_j c_pre) = -2 (s_j / cos_j) kappa to its derivative. So the reverse sweep
//     needs the pairs' logged values, one coefficient checkpoint per window, and no record per term and gate.
// The pairs are sorted once by sector (mpx_window.cuh: a term and its partner share a coset, so blocks never
// meet), and a block runs its sector's gates of a window with block barriers only.
#pragma once

#include "mpx_replay.h"
#include "mpx_window.cuh"

namespace mpx {

__global__ void __launch_bounds__(256) k_replay_tables(const GateDesc *__restrict__ gates, uint32_t L, int W, ReplayPlan p,
                                                        WindowTables *tables) {
    __shared__ TableWork s;
    const uint32_t lo = blockIdx.x * p.gates;
    window_tables(gates, L, lo, static_cast<int>(min(p.gates, L - lo)), W, tables[blockIdx.x],
                  p.comm + static_cast<uint64_t>(blockIdx.x) * kWindow, s);
}

// The gate (within the window) of pair r: the last whose first pair is at or before it.
__device__ __forceinline__ uint32_t gate_of(const uint64_t *s_begin, uint32_t n, uint64_t r) {
    uint32_t a = 0, b = n;
    while (b - a > 1) {
        const uint32_t m = (a + b) >> 1;
        if (s_begin[m] <= r) a = m;
        else b = m;
    }
    return a;
}

// Mask and sector of every pair of one window, and the pairs per (sector, gate). Bound by the emitters' key rows.
template <int W>
__global__ void __launch_bounds__(256) k_replay_count(const uint64_t *__restrict__ keys, ReplayPlan p, ReplaySort so,
                                                       uint32_t window, uint32_t L, const uint32_t *__restrict__ src,
                                                       const uint64_t *__restrict__ p_begin,
                                                       const unsigned long long *__restrict__ p_count, uint64_t first,
                                                       uint64_t count) {
    __shared__ uint64_t s_mask[64 * W], s_begin[kWindow], s_end[kWindow];
    __shared__ uint32_t s_inv[64 * W];
    const WindowTables &t = so.tables[window];
    const uint32_t lo = window * p.gates, n = min(p.gates, L - lo);
    for (uint32_t c = threadIdx.x; c < 64 * W; c += blockDim.x) {
        s_mask[c] = t.mask[c];
        s_inv[c] = t.inv[kLengths - 1][c];
    }
    if (threadIdx.x < n) {
        s_begin[threadIdx.x] = p_begin[lo + threadIdx.x];
        s_end[threadIdx.x] = p_begin[lo + threadIdx.x] + p_count[lo + threadIdx.x];
    }
    __syncthreads();
    uint32_t *seg = p.seg + static_cast<uint64_t>(window) * (p.sectors * p.gates + 1);
    for (uint64_t k = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; k < count;
         k += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t g = gate_of(s_begin, n, first + k);
        if (first + k >= s_end[g]) continue; // a place the log left empty
        uint64_t m[W];
        load_key<W>(keys, src[first + k], m);
        uint32_t f[1];
        so.c_mask[first + k] = window_mask<W, 1>(m, s_mask, s_inv, t.odd, f);
        const uint32_t s = static_cast<uint32_t>(mix64(f[0]) % p.sectors);
        so.c_sector[first + k] = static_cast<uint16_t>(s);
        atomicAdd(&seg[s * p.gates + g], 1u);
    }
}

// Counts to first pairs (exclusive prefix), one block per window, and the busiest sector's pairs; base: pairs of the
// windows before it.
__global__ void __launch_bounds__(1024) k_replay_prefix(ReplayPlan p, ReplaySort so) {
    __shared__ uint32_t s_part[32], s_most;
    if (threadIdx.x == 0) s_most = 0;
    const uint32_t n = p.sectors * p.gates;
    uint32_t *seg = p.seg + static_cast<uint64_t>(blockIdx.x) * (n + 1);
    uint32_t *cursor = so.cursor + static_cast<uint64_t>(blockIdx.x) * n;
    const uint32_t per = (n + blockDim.x - 1) / blockDim.x, lo = threadIdx.x * per, hi = min(n, lo + per);
    uint32_t sum = 0;
    for (uint32_t k = lo; k < hi; ++k) sum += seg[k];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += x;
    }
    if (lane == 31) s_part[warp] = incl;
    __syncthreads();
    uint32_t acc = so.base[blockIdx.x] + incl - sum;
    for (int w = 0; w < warp; ++w) acc += s_part[w];
    for (uint32_t k = lo; k < hi; ++k) {
        const uint32_t c = seg[k];
        seg[k] = acc;
        cursor[k] = acc;
        acc += c;
        if (k + 1 == n) seg[n] = acc;
    }
    __syncthreads();
    uint32_t most = 0;
    for (uint32_t k = threadIdx.x; k < p.sectors; k += blockDim.x) most = max(most, seg[(k + 1) * p.gates] - seg[k * p.gates]);
    most = __reduce_max_sync(0xFFFFFFFFu, most);
    if (lane == 0) atomicMax(&s_most, most);
    __syncthreads();
    if (threadIdx.x == 0) so.busiest[blockIdx.x] = s_most;
}

// Places the pairs (and their logged values) in any order within a sector and gate: the log of a propagation has none
// of its own.
__global__ void __launch_bounds__(256) k_replay_scatter(ReplayPlan p, ReplaySort so, uint32_t window, uint32_t L,
                                                         const uint32_t *__restrict__ src, const uint32_t *__restrict__ tgt,
                                                         const int8_t *__restrict__ code, const double *__restrict__ in_vs,
                                                         const double *__restrict__ in_vt, double *__restrict__ vs,
                                                         double *__restrict__ vt, const uint64_t *__restrict__ p_begin,
                                                         const unsigned long long *__restrict__ p_count, uint64_t first,
                                                         uint64_t count) {
    __shared__ uint64_t s_begin[kWindow], s_end[kWindow];
    const uint32_t lo = window * p.gates, n = min(p.gates, L - lo);
    if (threadIdx.x < n) {
        s_begin[threadIdx.x] = p_begin[lo + threadIdx.x];
        s_end[threadIdx.x] = p_begin[lo + threadIdx.x] + p_count[lo + threadIdx.x];
    }
    __syncthreads();
    uint32_t *cursor = so.cursor + static_cast<uint64_t>(window) * p.sectors * p.gates;
    for (uint64_t k = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; k < count;
         k += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint64_t r = first + k;
        const uint32_t g = gate_of(s_begin, n, r);
        if (r >= s_end[g]) continue;
        const uint32_t at = atomicAdd(&cursor[so.c_sector[r] * p.gates + g], 1u);
        p.src[at] = src[r];
        p.tgt[at] = tgt[r];
        p.code[at] = code[r];
        p.mask[at] = so.c_mask[r];
        if (in_vs != nullptr) {
            vs[at] = in_vs[r];
            vt[at] = in_vt[r];
        }
    }
}

// The same in the log's order: a structure that is replayed again and again keeps one order of its pairs, whichever
// engine sorts it (a clone has the same log). A gate's pairs are dealt to blocks in contiguous parts of kPlacePairs
// (parts[b]: gate and first part of block b's gate), a part to warps in contiguous shares. Every warp has its own
// cursor per sector: it counts, the counts become first places (after the parts before, whose counts
// k_replay_tally left), and it places its share 32 pairs at a time, each pair after those of its sector that come
// before it. Bound by the scattered stores of 17 bytes a pair; the next 32 are loaded ahead. The first gradient over
// a new graph, sort included: 100 qubits (8 layers, 8e7 pairs) 35.1 ms, with one block per gate 43, in any order 33;
// 50 qubits 10.7, 11.8 and 10.3 ms.
constexpr int kPlaceWarps = 16;

// Pairs per sector of every part that is not its gate's only or last one.
__global__ void __launch_bounds__(256) k_replay_tally(uint32_t sectors, ReplaySort so, const uint2 *__restrict__ parts,
                                                       const uint64_t *__restrict__ p_begin,
                                                       const unsigned long long *__restrict__ p_count) {
    __shared__ uint32_t s_count[kMaxSectors];
    const uint2 part = parts[blockIdx.x];
    const uint64_t lo = static_cast<uint64_t>(blockIdx.x - part.y) * kPlacePairs, first = p_begin[part.x] + lo;
    if (p_count[part.x] <= lo + kPlacePairs) return;
    for (uint32_t s = threadIdx.x; s < sectors; s += blockDim.x) s_count[s] = 0;
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < kPlacePairs; k += blockDim.x) atomicAdd(&s_count[so.c_sector[first + k]], 1u);
    __syncthreads();
    for (uint32_t s = threadIdx.x; s < sectors; s += blockDim.x) so.tally[static_cast<uint64_t>(blockIdx.x) * sectors + s] = s_count[s];
}

__global__ void __launch_bounds__(kPlaceWarps * 32)
    k_replay_place(ReplayPlan p, ReplaySort so, const uint2 *__restrict__ parts, const uint32_t *__restrict__ src,
                   const uint32_t *__restrict__ tgt, const int8_t *__restrict__ code, const uint64_t *__restrict__ p_begin,
                   const unsigned long long *__restrict__ p_count) {
    extern __shared__ uint32_t s_at[]; // [kPlaceWarps][sectors]
    const uint2 part = parts[blockIdx.x];
    const uint32_t window = part.x / p.gates, g = part.x % p.gates, S = p.sectors;
    const uint64_t skip = static_cast<uint64_t>(blockIdx.x - part.y) * kPlacePairs, all = p_count[part.x];
    if (all <= skip) return;
    const uint64_t first = p_begin[part.x] + skip, count = min(all - skip, uint64_t(kPlacePairs));
    for (uint32_t k = threadIdx.x; k < kPlaceWarps * S; k += blockDim.x) s_at[k] = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t share = ((count + kPlaceWarps - 1) / kPlaceWarps + 31) / 32 * 32;
    const uint64_t lo = min(count, warp * share), hi = min(count, lo + share);
    uint32_t *at = s_at + warp * S;
    for (uint64_t k = lo + lane; k < hi; k += 32) atomicAdd(&at[so.c_sector[first + k]], 1u);
    __syncthreads();
    const uint32_t *cursor = so.cursor + static_cast<uint64_t>(window) * S * p.gates;
    for (uint32_t s = threadIdx.x; s < S; s += blockDim.x) {
        uint32_t acc = cursor[s * p.gates + g];
        for (uint32_t b = part.y; b < blockIdx.x; ++b) acc += so.tally[static_cast<uint64_t>(b) * S + s];
        for (int w = 0; w < kPlaceWarps; ++w) {
            const uint32_t c = s_at[w * S + s];
            s_at[w * S + s] = acc;
            acc += c;
        }
    }
    __syncthreads();
    struct Pair {
        uint32_t sector, s, t;
        int8_t code;
        uint64_t mask;
    };
    auto load = [&](uint64_t k) {
        const uint64_t r = first + k;
        return k < hi ? Pair{so.c_sector[r], src[r], tgt[r], code[r], so.c_mask[r]} : Pair{kNoSector, 0, 0, 0, 0};
    };
    Pair next = load(lo + lane);
    for (uint64_t k = lo + lane; k - lane < hi; k += 32) { // warp-uniform
        const Pair q = next;
        next = load(k + 32);
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, q.sector), rank = __popc(peers & ((1u << lane) - 1u));
        uint32_t place = 0;
        if (k < hi) place = at[q.sector] + rank;
        __syncwarp();
        if (k < hi && rank == 0) at[q.sector] = place + __popc(peers);
        __syncwarp();
        if (k < hi) {
            p.src[place] = q.s;
            p.tgt[place] = q.t;
            p.code[place] = q.code;
            p.mask[place] = q.mask;
        }
    }
}

// c times the cos of the gates in m, first to last (the rounding of gate-by-gate scaling)
__device__ __forceinline__ double times_cos(double c, uint64_t m, const double *cos) {
    for (; m != 0; m &= m - 1) c *= cos[__ffsll(static_cast<long long>(m)) - 1];
    return c;
}
__device__ __forceinline__ double pair_phase(int8_t code) { return static_cast<double>(static_cast<int8_t>(code << 4) >> 4); }

// The pairs of one window, one sector per block. last[i]: the gates of the window already applied to term i.
// Bound by latency: per gate the two coefficients' loads and a block barrier; the next gate's pairs are loaded
// before the barrier. (Pairs two gates ahead with their coefficients prefetched to L2 one gate ahead were slower:
// 6x6 Hubbard loop 3.23 -> 3.78 ms.)
__global__ void __launch_bounds__(kSectorThreads, kSectorsPerSM)
    k_replay_pairs(double *__restrict__ coef, uint8_t *__restrict__ last, const uint32_t *__restrict__ longb, ReplayPlan p, uint32_t window,
                   const GateDesc *__restrict__ gates, uint32_t L, double *__restrict__ vs_log, double *__restrict__ vt_log) {
    __shared__ double s_cos[kWindow], s_sin[kWindow];
    __shared__ uint64_t s_comm[kWindow];
    __shared__ uint32_t s_seg[kWindow + 1];
    const uint32_t lo = window * p.gates, n = min(p.gates, L - lo), tid = threadIdx.x, T = blockDim.x;
    const uint32_t *seg = p.seg + static_cast<uint64_t>(window) * (p.sectors * p.gates + 1) + blockIdx.x * p.gates;
    if (seg[0] == seg[p.gates]) return;
    for (uint32_t g = tid; g <= n; g += T) {
        s_seg[g] = seg[g];
        if (g < n) {
            const GateDesc &gd = gates[L - 1 - (lo + g)];
            s_cos[g] = gd.cosv;
            s_sin[g] = gd.sinv;
            s_comm[g] = p.comm[static_cast<uint64_t>(window) * kWindow + g];
        }
    }
    __syncthreads();
    struct Pair {
        uint32_t s, t;
        int8_t code;
        uint64_t mask;
    };
    auto load = [&](uint32_t k) { return Pair{p.src[k], p.tgt[k], p.code[k], p.mask[k]}; };
    Pair next{};
    if (s_seg[0] + tid < s_seg[1]) next = load(s_seg[0] + tid);
    for (uint32_t g = 0; g < n; ++g) {
        const uint32_t b = s_seg[g], e = s_seg[g + 1];
        const Pair here = next;
        if (g + 1 < n && e + tid < s_seg[g + 2]) next = load(e + tid);
        if (b == e) continue; // block-uniform
        const double C = s_cos[g], S = s_sin[g];
        const uint64_t below = first_gates(g);
        for (uint32_t k = b + tid; k < e; k += T) {
            const Pair q = k == b + tid ? here : load(k);
            const double phi = pair_phase(q.code);
            double vs = coef[q.s], vt = coef[q.t];
            const uint32_t as = last[q.s], at = last[q.t];
            vs = times_cos(vs, q.mask & below & ~first_gates(as), s_cos);
            // an appended partner's slot holds the value the replay started it from until this gate; a partner
            // outside the only_rotate_len_k set is never scaled
            const bool appended = (q.code & 0x10) != 0;
            const bool unscaled = longb != nullptr && !appended && ((longb[q.t >> 5] >> (q.t & 31)) & 1u) != 0;
            if (!appended && !unscaled) vt = times_cos(vt, (q.mask ^ s_comm[g]) & below & ~first_gates(at), s_cos);
            coef[q.s] = C * vs - S * phi * vt;
            coef[q.t] = (unscaled ? vt : C * vt) + S * phi * vs;
            last[q.s] = static_cast<uint8_t>(g + 1);
            last[q.t] = static_cast<uint8_t>(g + 1);
            if (vs_log != nullptr) {
                vs_log[k] = vs;
                vt_log[k] = vt;
            }
        }
        __syncthreads();
    }
}

// ----- the dense passes ---------------------------------------------------------------------------------------

// What both dense passes share: the window's cos and first fold columns in shared memory, and per warp the
// anticommutation words of its 8 column words (gate-major, padded).
struct DenseShared {
    uint32_t word[kCloseWarps][kWindow * kClosePitch];
    double cos[kWindow];
    const uint32_t *col[kWindow][4]; // nullptr past the last
    uint8_t more[kWindow];           // 1: the gate has further columns (or the parity column)
};
__device__ __forceinline__ void dense_setup(DenseShared &s, const Store &st, const GateDesc *__restrict__ gates, uint32_t L,
                                            uint32_t lo, uint32_t n) {
    if (threadIdx.x < n) {
        const GateDesc &gd = gates[L - 1 - (lo + threadIdx.x)];
        s.cos[threadIdx.x] = gd.cosv;
        const int nf = gd.empty || gd.n_fold > kMaxFoldCols ? 0 : gd.n_fold;
        s.more[threadIdx.x] = gd.n_fold > 4 || gd.g_odd != 0;
#pragma unroll
        for (int f = 0; f < 4; ++f)
            s.col[threadIdx.x][f] = f < nf ? st.cols + static_cast<uint64_t>(gd.fold_cols[f]) * st.cstride : nullptr;
    }
    __syncthreads();
}
// The anticommutation words of column words [j0, j0 + 8) for the window's n gates (bits of terms >= n_terms, and of
// those in longb, zero).
__device__ __forceinline__ void dense_words(uint32_t *sw, const DenseShared &s, const Store &st, const GateDesc *__restrict__ gates,
                                            uint32_t L, uint32_t lo, uint32_t n, uint32_t parity_col, uint32_t j0,
                                            uint64_t n_terms, const uint32_t *__restrict__ longb) {
    const int lane = threadIdx.x & 31, w = lane & 7;
    const uint32_t j = j0 + w, nw = static_cast<uint32_t>((n_terms + 31) >> 5);
    uint32_t kept = j < nw && longb != nullptr ? ~longb[j] : 0xFFFFFFFFu;
    if (j == nw - 1 && (n_terms & 31) != 0) kept &= (1u << (n_terms & 31)) - 1u;
    for (uint32_t g0 = 0; g0 < n; g0 += 16) {
        uint32_t anti[4] = {0, 0, 0, 0};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const uint32_t g = g0 + 4 * h + (lane >> 3);
            if (g >= n || j >= nw) continue;
            uint32_t v[4];
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                const uint32_t *col = s.col[g][f];
                v[f] = col != nullptr ? col[j] : 0u;
            }
            anti[h] = v[0] ^ v[1] ^ v[2] ^ v[3];
            if (s.more[g]) anti[h] ^= more_columns(gates[L - 1 - (lo + g)], st, parity_col, j);
            anti[h] &= kept;
        }
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const uint32_t g = g0 + 4 * h + (lane >> 3);
            if (g < kWindow) sw[g * kClosePitch + w] = anti[h];
        }
    }
    __syncwarp();
}

// The end of a forward window: every term's remaining cos factors (its gates from last[i] on), last back to 0.
__global__ void __launch_bounds__(kCloseWarps * 32, 4)
    k_replay_close(Store st, uint32_t parity_col, const uint32_t *__restrict__ longb, uint8_t *__restrict__ last, const GateDesc *__restrict__ gates, uint32_t L,
                   uint32_t lo, uint32_t n, uint64_t n_terms, double *__restrict__ ck) {
    __shared__ __align__(16) DenseShared s;
    dense_setup(s, st, gates, L, lo, n);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *sw = s.word[warp];
    const uint32_t n_units = static_cast<uint32_t>((n_terms + 32 * kCloseWords - 1) / (32 * kCloseWords));
    for (uint32_t u = blockIdx.x * kCloseWarps + warp; u < n_units; u += gridDim.x * kCloseWarps) {
        const uint32_t j0 = u * kCloseWords;
        double c[kCloseWords];
        uint8_t from[kCloseWords];
#pragma unroll
        for (int w = 0; w < kCloseWords; ++w) {
            const uint64_t i = static_cast<uint64_t>(j0 + w) * 32 + lane;
            c[w] = i < n_terms ? st.coef[i] : 0.0;
            from[w] = i < n_terms ? last[i] : 0;
        }
        dense_words(sw, s, st, gates, L, lo, n, parity_col, j0, n_terms, longb);
#pragma unroll
        for (int w = 0; w < kCloseWords; ++w) {
            const uint64_t i = static_cast<uint64_t>(j0 + w) * 32 + lane;
            uint32_t m0 = transpose32(lane < n ? sw[lane * kClosePitch + w] : 0u, lane), m1 = 0;
            if (n > 32) m1 = transpose32(lane + 32 < n ? sw[(lane + 32) * kClosePitch + w] : 0u, lane);
            if (from[w] != 0) {
                const uint64_t rest = ~first_gates(from[w]);
                m0 &= static_cast<uint32_t>(rest);
                m1 &= static_cast<uint32_t>(rest >> 32);
                last[i] = 0;
            }
            if ((m0 | m1) != 0) {
                double x = c[w];
                for (; m0 != 0; m0 &= m0 - 1) x *= s.cos[__ffs(static_cast<int>(m0)) - 1];
                for (; m1 != 0; m1 &= m1 - 1) x *= s.cos[__ffs(static_cast<int>(m1)) + 31];
                c[w] = x;
                st.coef[i] = x;
            }
            if (ck != nullptr && i < n_terms) ck[i] = c[w];
        }
        __syncwarp();
    }
}

// acc0 / acc1 of lane j gain the sum over the lanes t with bit j / bit 32 + j of their mask set of kappa_t (whole
// warp). a0, a1: the masks transposed; kap: 32 doubles of the warp's own. Few bits per lane: one turn per bit of
// the fullest lane (about 20 instructions). More (terms that were appended together anticommute together): all 32
// terms in turn, 5 instructions each.
__device__ __forceinline__ void gather_kappa(uint32_t a0, uint32_t a1, double kappa, double *kap, double &acc0, double &acc1) {
    const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, max(__popc(a0), __popc(a1)));
    if (most == 0) return;
    if (most <= 6) {
        for (uint32_t k = 0; k < most; ++k) {
            const double k0 = __shfl_sync(0xFFFFFFFFu, kappa, a0 != 0 ? __ffs(static_cast<int>(a0)) - 1 : 0);
            if (a0 != 0) acc0 += k0;
            a0 &= a0 - 1;
            const double k1 = __shfl_sync(0xFFFFFFFFu, kappa, a1 != 0 ? __ffs(static_cast<int>(a1)) - 1 : 0);
            if (a1 != 0) acc1 += k1;
            a1 &= a1 - 1;
        }
        return;
    }
    kap[threadIdx.x & 31] = kappa;
    __syncwarp();
#pragma unroll
    for (int t = 0; t < 32; ++t) {
        const double k = kap[t];
        if (a0 & (1u << t)) acc0 += k;
        if (a1 & (1u << t)) acc1 += k;
    }
    __syncwarp();
}

// The block's share of the derivatives of the window's gates, to its slot of every gate's row: lane j's acc (times
// -2 tan) and direct parts of all warps, in order.
__device__ __forceinline__ void block_gradient(double (*s_sum)[kWindow], double acc0, double acc1, double d0, double d1,
                                               const GateDesc *__restrict__ gates, uint32_t L, uint32_t lo, uint32_t n,
                                               double *__restrict__ part, uint32_t slots, uint32_t slot) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t g = lane + 32 * h;
        if (g < n) {
            const GateDesc &gd = gates[L - 1 - (lo + g)];
            s_sum[warp][g] = (h ? d1 : d0) - 2.0 * (gd.sinv / gd.cosv) * (h ? acc1 : acc0);
        }
    }
    __syncthreads();
    for (uint32_t g = threadIdx.x; g < n; g += blockDim.x) {
        double t = 0.0;
        for (uint32_t w = 0; w < blockDim.x / 32; ++w) t += s_sum[w][g];
        part[static_cast<uint64_t>(g) * slots + slot] = t;
    }
}

// dE/dangle of the gates of blockIdx.y's window, one block per gate: the sum of its row's slots in a fixed order, so
// that the bits do not depend on which block came first. 14 values per thread, from L2; a launch for kSumWindows
// windows.
__global__ void __launch_bounds__(128) k_reverse_sum(ReplayPlan p, uint32_t window, uint32_t L, const double *__restrict__ part,
                                                      uint32_t slots, double *__restrict__ grad) {
    const uint32_t lo = (window + blockIdx.y) * p.gates, g = blockIdx.x;
    if (lo + g >= L) return;
    const double *row = part + (static_cast<uint64_t>(blockIdx.y) * kWindow + g) * slots;
    double t = 0.0;
    for (uint32_t k = threadIdx.x; k < slots; k += blockDim.x) t += row[k];
    __shared__ double s_part[4];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) grad[L - 1 - (lo + g)] = (s_part[0] + s_part[1]) + (s_part[2] + s_part[3]);
}

// The reverse sweep over one window's pairs, last gate first. event[i]: 0, or 1 + the earliest gate of the
// window met so far that pairs term i (from which on lam[i] is its adjoint before that gate).
__global__ void __launch_bounds__(kSectorThreads, kSectorsPerSM)
    k_reverse_pairs(double *__restrict__ lam, uint8_t *__restrict__ event, const uint32_t *__restrict__ longb, ReplayPlan p, uint32_t window,
                    const GateDesc *__restrict__ gates, uint32_t L, const double *__restrict__ vs_log,
                    const double *__restrict__ vt_log, double *__restrict__ part, uint32_t slots) {
    __shared__ double s_cos[kWindow], s_sin[kWindow];
    __shared__ uint64_t s_comm[kWindow];
    __shared__ uint32_t s_seg[kWindow + 1];
    __shared__ double s_sum[kSectorThreads / 32][kWindow], s_kap[kSectorThreads / 32][32];
    const uint32_t lo = window * p.gates, n = min(p.gates, L - lo), tid = threadIdx.x, T = blockDim.x;
    const uint32_t lane = tid & 31;
    const uint32_t *seg = p.seg + static_cast<uint64_t>(window) * (p.sectors * p.gates + 1) + blockIdx.x * p.gates;
    if (seg[0] == seg[p.gates]) {
        for (uint32_t g = tid; g < n; g += T) part[static_cast<uint64_t>(g) * slots + blockIdx.x] = 0.0;
        return;
    }
    for (uint32_t g = tid; g <= n; g += T) {
        s_seg[g] = seg[g];
        if (g < n) {
            const GateDesc &gd = gates[L - 1 - (lo + g)];
            s_cos[g] = gd.cosv;
            s_sin[g] = gd.sinv;
            s_comm[g] = p.comm[static_cast<uint64_t>(window) * kWindow + g];
        }
    }
    __syncthreads();
    struct Pair {
        uint32_t s, t;
        int8_t code;
        uint64_t mask;
        double vs, vt;
    };
    auto load = [&](uint32_t k) { return Pair{p.src[k], p.tgt[k], p.code[k], p.mask[k], vs_log[k], vt_log[k]}; };
    double acc0 = 0.0, acc1 = 0.0, d0 = 0.0, d1 = 0.0; // of gates lane and lane + 32
    Pair next{};
    if (s_seg[n - 1] + tid < s_seg[n]) next = load(s_seg[n - 1] + tid);
    for (uint32_t g = n; g-- > 0;) {
        const uint32_t b = s_seg[g], e = s_seg[g + 1];
        const Pair here = next;
        if (g > 0 && s_seg[g - 1] + tid < b) next = load(s_seg[g - 1] + tid);
        if (b == e) continue; // block-uniform
        const double C = s_cos[g], S = s_sin[g];
        const uint64_t above = ~first_gates(g + 1);
        for (uint32_t k0 = b; k0 < e; k0 += T) {
            if (k0 + (tid & ~31u) >= e) break; // warp-uniform
            const uint32_t k = k0 + tid;
            uint64_t ms = 0, mt = 0;
            double ks = 0.0, kt = 0.0, d = 0.0;
            if (k < e) {
                const Pair q = k0 == b ? here : load(k);
                const double phi = pair_phase(q.code);
                const uint32_t es = event[q.s], et = event[q.t];
                ms = q.mask & above;
                mt = (q.mask ^ s_comm[g]) & above;
                if (es != 0) ms &= first_gates(es - 1);
                if (et != 0) mt &= first_gates(et - 1);
                const bool appended = (q.code & 0x10) != 0;
                const bool out = longb != nullptr && ((longb[q.t >> 5] >> (q.t & 31)) & 1u) != 0; // never scaled
                if (out) mt = 0;
                // adjoints after gate g, and kappa of the stretches up to the pairs after it
                const double ls = times_cos(lam[q.s], ms, s_cos), lt = times_cos(lam[q.t], mt, s_cos);
                ks = (C * q.vs - S * phi * q.vt) * ls;
                kt = (C * q.vt + S * phi * q.vs) * lt;
                d = ls * (-2.0 * S * q.vs - 2.0 * C * phi * q.vt) +
                    lt * ((out && !appended ? 0.0 : -2.0 * S * q.vt) + 2.0 * C * phi * q.vs);
                lam[q.s] = C * ls + S * phi * lt;
                event[q.s] = static_cast<uint8_t>(g + 1);
                if (!appended) {
                    lam[q.t] = (out ? lt : C * lt) - S * phi * ls;
                    event[q.t] = static_cast<uint8_t>(g + 1);
                }
            }
            gather_kappa(transpose32(static_cast<uint32_t>(ms), lane), transpose32(static_cast<uint32_t>(ms >> 32), lane), ks, s_kap[tid >> 5], acc0, acc1);
            gather_kappa(transpose32(static_cast<uint32_t>(mt), lane), transpose32(static_cast<uint32_t>(mt >> 32), lane), kt, s_kap[tid >> 5], acc0, acc1);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xFFFFFFFFu, d, o);
            if (lane == (g & 31)) {
                if (g < 32) d0 += d;
                else d1 += d;
            }
        }
        __syncthreads();
    }
    block_gradient(s_sum, acc0, acc1, d0, d1, gates, L, lo, n, part, slots, blockIdx.x);
}

// The rest of a reverse window: every term's gates before its first pair (all of them for an unpaired term), for
// the n_terms terms the window began with. ck: their coefficients then; event back to 0.
__global__ void __launch_bounds__(kCloseWarps * 32, 3)
    k_reverse_close(Store st, uint32_t parity_col, const uint32_t *__restrict__ longb, double *__restrict__ lam, uint8_t *__restrict__ event,
                    const double *__restrict__ ck, const GateDesc *__restrict__ gates, uint32_t L, uint32_t lo, uint32_t n,
                    uint64_t n_terms, double *__restrict__ part, uint32_t slots, uint32_t first_slot) {
    __shared__ __align__(16) DenseShared s;
    __shared__ double s_sum[kCloseWarps][kWindow], s_kap[kCloseWarps][32];
    dense_setup(s, st, gates, L, lo, n);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *sw = s.word[warp];
    const uint32_t n_units = static_cast<uint32_t>((n_terms + 32 * kCloseWords - 1) / (32 * kCloseWords));
    double acc0 = 0.0, acc1 = 0.0;
    for (uint32_t u = blockIdx.x * kCloseWarps + warp; u < n_units; u += gridDim.x * kCloseWarps) {
        const uint32_t j0 = u * kCloseWords;
        double l[kCloseWords], c[kCloseWords];
        uint8_t ev[kCloseWords];
#pragma unroll
        for (int w = 0; w < kCloseWords; ++w) {
            const uint64_t i = static_cast<uint64_t>(j0 + w) * 32 + lane;
            l[w] = i < n_terms ? lam[i] : 0.0;
            c[w] = i < n_terms ? ck[i] : 0.0;
            ev[w] = i < n_terms ? event[i] : 0;
        }
        dense_words(sw, s, st, gates, L, lo, n, parity_col, j0, n_terms, longb);
#pragma unroll
        for (int w = 0; w < kCloseWords; ++w) {
            const uint64_t i = static_cast<uint64_t>(j0 + w) * 32 + lane;
            uint32_t a0 = lane < n ? sw[lane * kClosePitch + w] : 0u, a1 = n > 32 && lane + 32 < n ? sw[(lane + 32) * kClosePitch + w] : 0u;
            uint32_t m0 = transpose32(a0, lane), m1 = n > 32 ? transpose32(a1, lane) : 0u;
            if (__any_sync(0xFFFFFFFFu, ev[w] != 0)) {
                if (ev[w] != 0) {
                    const uint64_t before = first_gates(ev[w] - 1u);
                    m0 &= static_cast<uint32_t>(before);
                    m1 &= static_cast<uint32_t>(before >> 32);
                    event[i] = 0;
                }
                a0 = transpose32(m0, lane);
                a1 = n > 32 ? transpose32(m1, lane) : 0u;
            }
            double x = l[w];
            if ((m0 | m1) != 0 && x != 0.0) {
                for (; m0 != 0; m0 &= m0 - 1) x *= s.cos[__ffs(static_cast<int>(m0)) - 1];
                for (; m1 != 0; m1 &= m1 - 1) x *= s.cos[__ffs(static_cast<int>(m1)) + 31];
                lam[i] = x;
            }
            gather_kappa(a0, a1, c[w] * x, s_kap[warp], acc0, acc1);
        }
        __syncwarp();
    }
    block_gradient(s_sum, acc0, acc1, 0.0, 0.0, gates, L, lo, n, part, slots, first_slot + blockIdx.x);
}

} // namespace mpx
