// mpx_replay.h -- host interface of the windowed replay of a frozen structure (mpx_replay.cuh).
#pragma once

#include "mpx_window.h"

namespace mpx {

// The pairs of a frozen structure in replay order: by window of `gates` steps, by sector, by gate. seg holds the
// first pair of every (sector, gate) of every window, and one past the last.
struct ReplayPlan {
    uint32_t gates, windows, sectors;
    uint32_t *src, *tgt; // emitter and partner
    int8_t *code;        // phase (+1 / -1 / 0) | 0x10 for an appended partner
    uint64_t *mask;      // the window's gates that anticommute with the emitter
    uint32_t *seg;       // [windows][sectors * gates + 1]
    uint64_t *comm;      // [windows][kWindow] anticommutation among the window's gates
};

struct ReplayLaunch {
    Store st;
    const uint32_t *longb; // one bit per term outside the only_rotate_len_k set (never scaled), or nullptr
    const GateDesc *desc;
    uint32_t L;
    int W;
    unsigned blocks; // grid of the dense passes
    cudaStream_t stream;
};

// Scratch of the sort: tables and cursors of all windows, and every pair's mask and sector.
struct ReplaySort {
    WindowTables *tables;
    uint32_t *cursor;   // [windows][sectors * gates]
    uint32_t *base;     // [windows] pairs of the windows before
    uint32_t *busiest;  // [windows] out: most pairs of one sector
    uint64_t *c_mask;
    uint16_t *c_sector;
    uint32_t *tally;    // [parts][sectors] (replay_place)
};
constexpr uint32_t kPlacePairs = 1u << 15; // pairs per part

cudaError_t replay_tables(const ReplayLaunch &a, const ReplayPlan &p, const ReplaySort &s);
cudaError_t replay_count(const ReplayLaunch &a, const ReplayPlan &p, const ReplaySort &s, uint32_t window,
                         const uint32_t *src, const uint64_t *p_begin, const unsigned long long *p_count, uint64_t first,
                         uint64_t count);
cudaError_t replay_prefix(const ReplayLaunch &a, const ReplayPlan &p, const ReplaySort &s);
cudaError_t replay_scatter(const ReplayLaunch &a, const ReplayPlan &p, const ReplaySort &s, uint32_t window,
                           const uint32_t *src, const uint32_t *tgt, const int8_t *code, const double *in_vs,
                           const double *in_vt, double *vs, double *vt, const uint64_t *p_begin,
                           const unsigned long long *p_count, uint64_t first, uint64_t count);

// The pairs in the log's order within a sector and gate. parts: [n_parts] the gate of every part and the gate's first part.
cudaError_t replay_place(const ReplayLaunch &a, const ReplayPlan &p, const ReplaySort &s, const uint2 *parts, uint32_t n_parts,
                         const uint32_t *src, const uint32_t *tgt, const int8_t *code, const uint64_t *p_begin,
                         const unsigned long long *p_count);

// One window forward: its pairs (vs, vt: logged when not null), then the dense pass over the n_end terms it
// leaves; ck: the coefficients after the window, when not null. last: [terms] zero between windows.
cudaError_t replay_forward(const ReplayLaunch &a, const ReplayPlan &p, uint32_t window, uint64_t n_end, uint8_t *last,
                           double *vs, double *vt, double *ck);
// One window backward: its pairs, then the dense pass over the n_start terms it began with (ck: their
// coefficients then). Every block's share of dE/dangle goes to its slot of part, [kSumWindows][kWindow][replay_slots]
// by window mod kSumWindows; the window 0 and every kSumWindows-th also adds the slots up to grad.
constexpr uint32_t kSumWindows = 8;
inline uint32_t replay_slots(const ReplayLaunch &a, const ReplayPlan &p) { return p.sectors + a.blocks; }
cudaError_t replay_reverse(const ReplayLaunch &a, const ReplayPlan &p, uint32_t window, uint64_t n_start, double *lam,
                           uint8_t *event, const double *vs, const double *vt, const double *ck, double *part, double *grad);

}  // namespace mpx
