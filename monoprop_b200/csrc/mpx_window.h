// mpx_window.h -- host interface of the window kernels (mpx_window.cuh) for the engine.
#pragma once

#include <cuda_runtime.h>

#include "mpx_device.cuh"

namespace mpx {

constexpr int kWindow = 64;             // gates per window at most (the masks are 64-bit words)
constexpr uint32_t kChunk = 1024;       // list slots per chunk of a sector's list
constexpr uint32_t kSectorChunks = 512; // chunks per sector at most
// A sector's list may grow to this many chunks, eight times the mean sector's at the window's start or four times its
// own then, whichever is most; a window in which one grows past that is given up and its gates run one by one. One
// block has all the terms of a coset, at some 0.05 us each per gate: without a limit a few terms that grow to 1e6 within
// the window (150 gates on 10 of 161 modes) kept it for 180 ms, 9 ms gate by gate; 4096 terms take 1 ms at most.
constexpr uint32_t kGrowChunks = 4;
constexpr uint32_t kMaxSectors = 2048;
// A window runs only while at most half of the store's terms are candidates (a quarter above kLargeTerms terms).
// With more, leaving the others aside gains less than the lists cost, and both paths are bound by the emitted
// branches' scattered accesses: the 5x10 kicked Ising circuit of 12 layers (3e7 terms, a third of them active)
// takes 114 ms in windows and 104 ms gate by gate, the Schrodinger picture of the 20-qubit line (4.5e6 terms, all
// active) 4.8 and 3.8 ms, the 10x10 circuit (7 % active in the end, 40 % at 2e6 terms) 93 and 179 ms, and 101 ms
// with a quarter from the start. Up to some 1e4 terms a gate is bound by its launches, and windows win at any
// density (5x3 Hubbard lattice, 6e4 terms: 4.5 ms against 6.2 ms).
constexpr uint64_t kDenseTerms = uint64_t(1) << 16, kLargeTerms = uint64_t(1) << 22;
constexpr uint64_t kDenseGates = 192;   // steps taken gate by gate before the next try
// Fewer steps than this run gate by gate without a try: over 32 gates windows take 1.2 to 1.4 times as long, a try that
// is declined some 0.1 ms (8 gates: 0.09 ms gate by gate, 0.19 with a try), over 64 gates 0.8 times.
constexpr uint64_t kLeastGates = 32;
constexpr int kLengths = 4;             // window lengths tried: kWindow / 8, / 4, / 2 and kWindow gates
constexpr int kSectorThreads = 128;     // threads of a sector's block
constexpr int kSectorsPerSM = 8;        // resident blocks per SM it is compiled for; one wave of sectors

// The i-th window length tried, of at most `most` gates.
__host__ __device__ inline uint32_t window_length(int i, uint32_t most) {
    const uint32_t n = static_cast<uint32_t>(kWindow) >> (kLengths - 1 - i);
    return n < most ? n : most;
}

// Linear maps of a key for the next window: the XOR over its set bits of
struct WindowTables {
    uint64_t mask[64 * kMaxWords];          // the gates whose fold holds the bit (anticommutation),
    uint32_t inv[kLengths][64 * kMaxWords]; // the bit's value of f, zero on the generators of the i-th length
    uint64_t odd;        // Majorana gates of odd length (anticommute with the other odd terms)
    double sin[kWindow]; // |sin| of the gates
};

// Device state of the running window. count/scatter write it, gates and commit update it, the next close reads it.
struct WindowCtl {
    uint32_t n_cand;   // candidates collected for the next window
    uint32_t n_chunks; // chunks of the pool in use
    uint32_t lo;       // first step of the last window
    uint32_t gates;    // its number of gates
    uint32_t run;      // 1: the window runs (0: an earlier window stalled, its kernels do nothing)
    uint32_t overflow; // 1: the appends did not fit, 2: a sector's list or all of them together are full (nothing is committed then),
                       // 3: too many active terms or too dear, the window does not run
    uint32_t pending;  // 1: its passive terms still lack their cos factors, its counters their place
    uint32_t grow;     // chunks a sector's list may grow to (kGrowChunks)
    uint64_t n_start;  // store size at its start
    uint64_t comm[kWindow];   // bit j of entry b: gates b and j of the window anticommute
    WindowTables tables;
    uint32_t anti[kWindow];     // per gate: anticommuting terms among the window's appends,
    uint32_t emitted[kWindow];  //           emitted branches,
    uint32_t appended[kWindow]; //           appends
    uint32_t load[kLengths][kMaxSectors]; // anticommuting gates of each sector's sampled terms, by window length
    uint32_t sector[kMaxSectors];         // list entries per sector at the start
    uint32_t filled[kMaxSectors];         // of them placed so far (scatter)
};

// The active terms' lists. Slot s belongs to chunk s / kChunk; a chunk belongs to one sector.
struct WindowScratch {
    double *a_val;      // [slots] current coefficient
    uint64_t *a_mask;   // [slots] gates of the window the term anticommutes with
    uint32_t *a_idx;    // [slots] term
    uint32_t *a_bits;   // [chunks][kWindow][kChunk / 32] the masks by gate, one bit per slot
    uint8_t *a_lead;    // [slots] 1 + the last gate at which the term emitted as a leader
    uint32_t *fill;     // [chunks] slots in use
    uint32_t *slot_of;  // [cap] list slot of an active term
    uint32_t *act;      // [ceil(cap / 32)] one bit per term below n_start: on a list
    uint32_t *q_tgt;    // [slots] partner of a queued branch beyond the shared-memory queue
    uint64_t slots;     // a multiple of kChunk
    WindowCtl *ctl;
};
constexpr uint16_t kNoSector = 0xFFFF;

// What every launch of a window takes: the store, the engine's scratch and settings, the uploaded circuit.
struct WindowLaunch {
    Store st;
    Scratch sc;
    WindowScratch ws;
    Counters *cnt;
    const GateDesc *gates;
    uint32_t L;
    Trunc tr;
    uint64_t *stats;
    int W, basis;
    uint32_t sectors, threads; // blocks of the gates kernel and their threads
    unsigned blocks;           // grid of the other kernels
    cudaStream_t stream;
};

// The dense pass: applies the last window's pending cos factors and collects the candidates of the next window
// (of the steps from cnt->step on and before hi; none when there are none).
cudaError_t window_close(const WindowLaunch &a, uint32_t hi);
// The next window of gates before step hi (from cnt->step on; how many is decided on the device), in five
// launches: sample, count, scatter, gates, commit.
cudaError_t window_gates(const WindowLaunch &a, uint32_t hi);

// The dense pass after the last window of a stretch; nothing is pending afterwards.
cudaError_t window_finish(const WindowLaunch &a);
// In a captured sequence: goes on at step `next` if the windows have ended at step `at`, else stops it.
cudaError_t window_handover(const WindowLaunch &a, uint32_t at, uint32_t next);

}  // namespace mpx
