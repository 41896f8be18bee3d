// mpx_window.cu -- launchers of the window kernels (mpx_window.cuh), one variant per key width, basis and
// basis_change. A translation unit of its own: it compiles beside the engine's.
#include <algorithm>

#include "mpx_replay.cuh"
#include "mpx_window.cuh"

namespace mpx {
namespace {

template <int W, int B, bool MAPPED>
cudaError_t sectors_launch(const WindowLaunch &a) {
    const auto kernel = &k_window_gates<W, B, MAPPED>;
    const size_t bytes = sizeof(GateShared<W>) + gate_lists_bytes(a.threads);
    // the attribute belongs to the function and the device; setting it is cheap next to the window it runs
    const cudaError_t ce = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    if (ce != cudaSuccess) return ce;
    kernel<<<a.sectors, a.threads, bytes, a.stream>>>(a.st, a.sc, a.ws, a.cnt, a.gates, a.L, a.tr);
    return cudaGetLastError();
}

template <int W>
cudaError_t gates_w(const WindowLaunch &a, uint32_t hi) {
    // the candidates' masks and sectors live where the queues and slot bits go later
    auto *c_mask = reinterpret_cast<uint64_t *>(a.sc.q_val);
    auto *c_sector = reinterpret_cast<uint16_t *>(a.ws.a_bits);
    k_window_sample<W><<<kSampleBlocks, 256, 0, a.stream>>>(a.st, a.ws, a.sc.q_src, a.cnt, hi, a.sectors, a.tr);
    k_window_count<W><<<a.blocks, 256, 0, a.stream>>>(a.st, a.ws, a.sc.q_src, c_mask, c_sector, a.cnt, hi, a.sectors, a.tr);
    k_window_scatter<<<a.blocks, 256, 0, a.stream>>>(a.st, a.ws, a.sc.q_src, c_mask, c_sector, a.cnt, hi, a.sectors);
    cudaError_t ce = cudaGetLastError();
    if (ce != cudaSuccess) return ce;
    if (a.basis == 1) ce = sectors_launch<W, 1, false>(a);
    else if (a.tr.basis_rows != nullptr) ce = sectors_launch<W, 0, true>(a);
    else ce = sectors_launch<W, 0, false>(a);
    if (ce != cudaSuccess) return ce;
    k_window_commit<W><<<a.blocks, kBlock, 0, a.stream>>>(a.st, a.ws, a.cnt);
    return cudaGetLastError();
}

}  // namespace

cudaError_t window_close(const WindowLaunch &a, uint32_t hi) {
    k_window_close<<<a.blocks + 1, kCloseWarps * 32, 0, a.stream>>>(a.st, 64u * a.W, a.ws, a.sc.q_src, a.cnt, a.gates, a.L,
                                                                hi, a.tr, a.stats);
    return cudaGetLastError();
}

cudaError_t window_handover(const WindowLaunch &a, uint32_t at, uint32_t next) {
    k_window_handover<<<1, 1, 0, a.stream>>>(a.cnt, at, next);
    return cudaGetLastError();
}

cudaError_t window_finish(const WindowLaunch &a) {
    const cudaError_t ce = window_close(a, 0);
    return ce != cudaSuccess ? ce : cudaMemsetAsync(&a.ws.ctl->pending, 0, sizeof(uint32_t), a.stream);
}

cudaError_t window_gates(const WindowLaunch &a, uint32_t hi) {
    switch (a.W) {
    case 1: return gates_w<1>(a, hi);
    case 2: return gates_w<2>(a, hi);
    case 3: return gates_w<3>(a, hi);
    case 4: return gates_w<4>(a, hi);
    case 5: return gates_w<5>(a, hi);
    case 6: return gates_w<6>(a, hi);
    case 7: return gates_w<7>(a, hi);
    default: return gates_w<8>(a, hi);
    }
}

// ----- replay of a frozen structure (mpx_replay.cuh) -----

namespace {
unsigned pair_blocks(uint64_t count) { return static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>((count + 255) / 256, 2368))); }

template <int W>
void count_w(const ReplayLaunch &a, const ReplayPlan &p, const ReplaySort &s, uint32_t window, const uint32_t *src,
             const uint64_t *p_begin, const unsigned long long *p_count, uint64_t first, uint64_t count) {
    k_replay_count<W><<<pair_blocks(count), 256, 0, a.stream>>>(a.st.keys, p, s, window, a.L, src, p_begin, p_count, first, count);
}
}  // namespace

cudaError_t replay_tables(const ReplayLaunch &a, const ReplayPlan &p, const ReplaySort &s) {
    k_replay_tables<<<p.windows, 256, 0, a.stream>>>(a.desc, a.L, a.W, p, s.tables);
    return cudaGetLastError();
}

cudaError_t replay_count(const ReplayLaunch &a, const ReplayPlan &p, const ReplaySort &s, uint32_t window,
                         const uint32_t *src, const uint64_t *p_begin, const unsigned long long *p_count, uint64_t first,
                         uint64_t count) {
    if (count == 0) return cudaSuccess;
    switch (a.W) {
    case 1: count_w<1>(a, p, s, window, src, p_begin, p_count, first, count); break;
    case 2: count_w<2>(a, p, s, window, src, p_begin, p_count, first, count); break;
    case 3: count_w<3>(a, p, s, window, src, p_begin, p_count, first, count); break;
    case 4: count_w<4>(a, p, s, window, src, p_begin, p_count, first, count); break;
    case 5: count_w<5>(a, p, s, window, src, p_begin, p_count, first, count); break;
    case 6: count_w<6>(a, p, s, window, src, p_begin, p_count, first, count); break;
    case 7: count_w<7>(a, p, s, window, src, p_begin, p_count, first, count); break;
    default: count_w<8>(a, p, s, window, src, p_begin, p_count, first, count); break;
    }
    return cudaGetLastError();
}

cudaError_t replay_prefix(const ReplayLaunch &a, const ReplayPlan &p, const ReplaySort &s) {
    k_replay_prefix<<<p.windows, 1024, 0, a.stream>>>(p, s);
    return cudaGetLastError();
}

cudaError_t replay_scatter(const ReplayLaunch &a, const ReplayPlan &p, const ReplaySort &s, uint32_t window,
                           const uint32_t *src, const uint32_t *tgt, const int8_t *code, const double *in_vs,
                           const double *in_vt, double *vs, double *vt, const uint64_t *p_begin,
                           const unsigned long long *p_count, uint64_t first, uint64_t count) {
    if (count == 0) return cudaSuccess;
    k_replay_scatter<<<pair_blocks(count), 256, 0, a.stream>>>(p, s, window, a.L, src, tgt, code, in_vs, in_vt, vs, vt,
                                                               p_begin, p_count, first, count);
    return cudaGetLastError();
}

cudaError_t replay_forward(const ReplayLaunch &a, const ReplayPlan &p, uint32_t window, uint64_t n_end, uint8_t *last,
                           double *vs, double *vt, double *ck) {
    const uint32_t lo = window * p.gates, n = std::min(p.gates, a.L - lo);
    k_replay_pairs<<<p.sectors, kSectorThreads, 0, a.stream>>>(a.st.coef, last, a.longb, p, window, a.desc, a.L, vs, vt);
    k_replay_close<<<a.blocks, kCloseWarps * 32, 0, a.stream>>>(a.st, 64u * a.W, a.longb, last, a.desc, a.L, lo, n,
                                                                n_end, ck);
    return cudaGetLastError();
}

cudaError_t replay_place(const ReplayLaunch &a, const ReplayPlan &p, const ReplaySort &s, const uint2 *parts, uint32_t n_parts,
                         const uint32_t *src, const uint32_t *tgt, const int8_t *code, const uint64_t *p_begin,
                         const unsigned long long *p_count) {
    if (n_parts == 0) return cudaSuccess;
    const size_t bytes = static_cast<size_t>(kPlaceWarps) * p.sectors * sizeof(uint32_t); // at most 128 KB (kMaxSectors)
    const cudaError_t ce = cudaFuncSetAttribute(k_replay_place, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    if (ce != cudaSuccess) return ce;
    k_replay_tally<<<n_parts, 256, 0, a.stream>>>(p.sectors, s, parts, p_begin, p_count);
    k_replay_place<<<n_parts, kPlaceWarps * 32, bytes, a.stream>>>(p, s, parts, src, tgt, code, p_begin, p_count);
    return cudaGetLastError();
}

cudaError_t replay_reverse(const ReplayLaunch &a, const ReplayPlan &p, uint32_t window, uint64_t n_start, double *lam,
                           uint8_t *event, const double *vs, const double *vt, const double *ck, double *part, double *grad) {
    const uint32_t lo = window * p.gates, n = std::min(p.gates, a.L - lo), slots = replay_slots(a, p), at = window % kSumWindows;
    double *row = part + static_cast<uint64_t>(at) * kWindow * slots;
    k_reverse_pairs<<<p.sectors, kSectorThreads, 0, a.stream>>>(lam, event, a.longb, p, window, a.desc, a.L, vs, vt, row, slots);
    k_reverse_close<<<a.blocks, kCloseWarps * 32, 0, a.stream>>>(a.st, 64u * a.W, a.longb, lam, event, ck, a.desc, a.L, lo, n,
                                                                 n_start, row, slots, p.sectors);
    if (at == 0) // windows come last to first
        k_reverse_sum<<<dim3(p.gates, std::min(kSumWindows, p.windows - window)), 128, 0, a.stream>>>(p, window, a.L, part, slots, grad);
    return cudaGetLastError();
}

}  // namespace mpx
