// ps_run.h -- a run of rotation layers on a small sum in one cooperative launch (ps_run.cu).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "ps_kernels.h"

namespace psb {

constexpr int kRunThreads = 512;
constexpr int kRunMaxBlocks = 256;
constexpr int kRunLevels = 4;     // partner delta bits of a layer the run takes
constexpr int kRunBins = 2048;    // TopN digit bins
constexpr int kRunCand = 1024;    // boundary-bin keys the select ranks directly
constexpr int kRunMaxLayers = 2048;

// One layer of a run's program (device memory): RotLayer's fields with one coefficient type.
template <int W, typename T>
struct alignas(16) RunLayer {
    uint64_t gx[W], gz[W];
    T a0[16], a1[16];
    double cos64, sin64;
    float cos32, sin32;
    int32_t wide, partners;
    int32_t qw[2], qb[2];
    uint32_t pattern_mask;
    int32_t nlev;
    uint32_t rank[kRunLevels];
    int32_t noise_first, noise_n;  // folded noise: its channels' place in the run's noise tables
    int32_t inner;                 // a permutation's step before its last: no keep program
    int32_t group;                 // steps of the permutation that starts here (they run or stop together)
};

// A block's part of a layer, read by every block after the layer's first barrier.
template <int W>
struct alignas(16) RunSummary {
    uint64_t first[2 * W], last[2 * W];               // its first and last emitting keys
    uint32_t rows, partners;
    uint16_t lstart[kRunLevels], lsplit[kRunLevels];  // last / first group start and split among its
    uint16_t fstart[kRunLevels], fsplit[kRunLevels];  // partners after the first one (0xFFFF: none)
};

// Control words of a run (zeroed before each launch).
struct alignas(16) RunState {
    unsigned int bar;
    unsigned int layers_done;
    unsigned int cand_n[3];
    unsigned int window;
    unsigned long long n;
    unsigned long long boundary;  // last TopN boundary (full-range select key)
    unsigned int ties[kRunMaxBlocks];
    alignas(16) unsigned int hist[3][kRunBins];  // read four bins at a time
    alignas(16) unsigned long long cand[2][kRunCand];
};

template <int W, typename T>
struct RunArgs {
    const uint64_t* Sk;  // input store, n rows (not written)
    const T* Sc;
    uint64_t n;
    uint64_t* Wk;        // work store: the run's rows between layers and its result; wcap rows
    T* Wc;
    uint64_t wcap;
    uint64_t* Pk;        // partners, pcap rows
    T* Pc;
    uint64_t pcap;
    const RunLayer<W, T>* prog;
    uint32_t nlayers;
    const T* noise_f;         // [channel][4]
    const uint16_t* noise_q;  // [channel]
    KeepProg keep;
    unsigned long long topn;  // 0: no TopN pass
    uint64_t window_base;     // with `window`: where the first digit's window starts
    int window;
    RunSummary<W>* sums;      // kRunMaxBlocks
    RunState* st;
    unsigned int* out_rows;   // per layer: rows before the pass, rows after it (both zeroed)
    unsigned int* after_rows;
    unsigned int* drops;      // per folded channel: own rows first dropped after it (zeroed)
    Ctl* ctl;
    uint32_t rcap;            // rows a block holds
};

template <int W, typename T>
struct RunOps {
    static uint32_t rows_per_block();  // 0: the device cannot run it
    static cudaError_t launch(const RunArgs<W, T>& a, int blocks, cudaStream_t st, KernelProf* prof);
};

}  // namespace psb
