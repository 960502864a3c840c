// ps_cut.h -- TopN without a compaction between rotation layers (ps_cut.cu).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "ps_kernels.h"

namespace psb {

constexpr int kCutThreads = 512;
constexpr int kCutLevels = 4;             // delta bits of a next layer the listing takes
// The cut's window of 2048 bins of |c|^2's bit pattern: 1024 bins of 1/1024 octave around the last
// boundary and 512 bins of 1/32 octave on either side (the boundary moves a tenth of an octave from
// layer to layer in the middle, several octaves once in a dozen layers of random angles).  All in
// the pattern's high word, so the merge bins a row in a few 32-bit operations.
constexpr int kCutFine = 42, kCutCoarse = 47;
constexpr uint32_t kCutSide = 512u << (kCutCoarse - 32);     // 16 octaves, in the high word
constexpr uint32_t kCutMid = 1024u << (kCutFine - 32);       // one
constexpr uint32_t kCutReach = kCutSide + kCutMid / 2;       // from the window's base to its middle
constexpr uint32_t kCutCand = 1u << 21;   // boundary-bin rows the select takes
constexpr uint32_t kCutBlockCand = 1024;  // of them a block gathers in shared memory
constexpr uint32_t kCutAllTies = 0xffffffffu;
// The window's base (high word) for the last boundary (a select key: a bit pattern plus one).
inline uint32_t cut_base(unsigned long long boundary) {
    const uint32_t hi = (uint32_t)((boundary - 1) >> 32) >> (kCutFine - 32) << (kCutFine - 32);
    return hi - kCutReach;
}
#ifdef __CUDACC__
// The bin of coefficient c (below the window and NaN 0, above it 2047: both mean it is outside).
template <typename T>
__device__ __forceinline__ uint32_t cut_bin(T c, uint32_t base) {
    const double v = (double)c, q = __dmul_rn(v, v);
    const uint32_t d = (uint32_t)__double2hiint(q) - base, m = d - kCutSide;
    uint32_t bin = (d >> (kCutCoarse - 32)) + (d >= kCutSide ? 992u : 0u);
    if (m < kCutMid) bin = 512u + (m >> (kCutFine - 32));
    if ((int32_t)d < 0 || !(q == q)) bin = 0u;
    return bin > 2047u ? 2047u : bin;
}
// Its lowest pattern and the bits below it.
__device__ __forceinline__ uint64_t cut_bin_low(uint32_t bin, uint32_t base, int& bits) {
    const bool mid = bin >= 512 && bin < 1536;
    bits = mid ? kCutFine : kCutCoarse;
    const uint32_t d = mid ? kCutSide + ((bin - 512) << (kCutFine - 32))
                           : (bin < 512 ? bin << (kCutCoarse - 32) : (bin - 992) << (kCutCoarse - 32));
    return (uint64_t)(base + d) << 32;
}
#endif

// Per merge tile, written by the cut: rows and partners before it within its block's run of tiles,
// its own partners, and the level scans' prefix (max, -1 none) and suffix (min, kCutNone) in
// positions within the block's run.
constexpr int kCutNone = 0x7fffffff;
struct CutTile {
    uint32_t rows_before, part_before, partners, flags;  // flags: first partner's starts | splits << 4
    int fwd[2 * kCutLevels], bwd[2 * kCutLevels];
};
// Per block of the cut: totals and aggregates of its run of tiles, then its place in the whole.
struct CutBlock {
    uint32_t rows, partners;
    uint32_t first_row, last_row, first_tile, pad;  // first / last emitting row, the first's tile
    int fwd[2 * kCutLevels], bwd[2 * kCutLevels];   // aggregates; after the last block: prefix, suffix
    uint32_t rbase, pbase;
};
// Results, read by the host after the pass.
struct CutState {
    unsigned int ticket;
    unsigned int status;          // 0: cut at `boundary`; otherwise nothing can be read from it
    unsigned int ncand;           // boundary-bin rows gathered
    unsigned int last_tie;        // the last row equal to the boundary that stays (kCutAllTies: all)
    unsigned long long boundary;  // full-range select key
    unsigned long long above;     // rows above it
    unsigned long long rows;      // rows the slots hold, dead ones among them
    unsigned long long partners;  // of them listed as emitting under the next layer
};

// The rows of a slotted store that a cut left in place: tile t's rows start at row t * slot_rows and
// pr[t] rows lie before it (pr[tiles] in all).
struct CutStore {
    const uint32_t* pr;
    uint32_t tiles, slot_rows;
};

// Which of those rows are live: |c|^2 above the boundary's, or equal to it and not after row last_tie
// (`at`: a row's place in the slots, or its rank among the rows with last_tie's rank given).  NaN is
// never live.
struct CutLive {
    double bound;
    uint32_t last_tie;
#ifdef __CUDACC__
    __device__ __forceinline__ bool operator()(double c, uint32_t at) const { return test(c, at, last_tie); }
    __device__ __forceinline__ bool test(double c, uint32_t at, const uint32_t& last) const {
        const double q = __dmul_rn(c, c);
        if (q == bound) return at <= last;  // rare
        return q > bound;
    }
#endif
};

template <int W, typename T>
struct CutArgs {
    const uint64_t* keys;   // the merge's slotted output
    const T* coef;
    const uint8_t* flags;   // the rows' partner tests under the next layer: flag_stride(slot_rows) a tile
    const unsigned int* count;
    uint32_t slot_rows;
    Levels next;            // the next layer's delta bits
    CutTile* tiles;
    CutBlock* blocks;
    uint16_t* plist;        // per tile, at its slot: the emitting rows (within the tile)
    uint16_t* D;            // and their divergence ranks from the one before
    unsigned int* hist;     // 2048 window bins of the merge's outputs; zeroed
    uint32_t base;          // the window's (cut_base)
    unsigned long long keep_n;
    uint64_t* cand;         // kCutCand patterns,
    uint32_t* cand_row;     // and their rows
    CutState* state;        // zeroed before the launch
    Ctl* ctl;
};

template <int W, typename T>
struct CutOps {
    // blocks of the cut (and runs of tiles)
    static int blocks(int sms);
    static cudaError_t configure();
    static cudaError_t cut(const CutArgs<W, T>& a, int sms, cudaStream_t st, KernelProf* prof);
    // The listed partners of a cut store at their sorted slots, and pr.
    static cudaError_t place(const CutArgs<W, T>& a, const RotLayer<W>& L, uint32_t tiles, CutLive live, uint64_t m, uint64_t* Pk, T* Pc, uint32_t* pr, int sms, cudaStream_t st, KernelProf* prof);
    // Merge-path split points of a cut store's rows and the partners: bounds[t], and the slot of its row
    // with the rows before that slot and to its end.
    static cudaError_t partition(const uint64_t* Sk, uint64_t n, const CutStore& S, const uint64_t* Pk, uint64_t m,
                                 uint32_t tile_items, ulonglong2* bounds, uint4* bslot, int sms, cudaStream_t st,
                                 KernelProf* prof);
};

}  // namespace psb
