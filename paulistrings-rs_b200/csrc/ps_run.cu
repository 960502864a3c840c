// ps_run.cu -- a run of rotation layers on a small sum in one cooperative launch.
//
// A sum of up to a few hundred thousand terms fits the multiprocessors' shared memory, and its
// layers are bound by latency, not by memory: the per-layer kernels (ps_rotation.cu, ps_store.cu)
// are eight or nine launches and a host round trip of a few microseconds each around passes that
// move a megabyte.  Here one block per multiprocessor keeps its slice of the sorted sum in
// shared memory from layer to layer, and a layer costs two grid barriers (four with a TopN
// selection), all bounded:
//
//   classify   the block's rows that emit a partner are listed; divergence ranks of neighbours and
//              the block's scans over them (the level scans of ps_rotation.cu) run in the block;
//              its row and partner counts, its edge keys and scan aggregates are published.
//   barrier
//   place      every block combines the published aggregates, so it knows its rows' positions and
//              each of its partners' sorted slots, and writes both to global memory (L2).
//   barrier
//   merge      the block takes an equal share of the merged order (merge-path split found by two
//              warps), loads it, and merges: each consumed row leaves its output at its merged
//              position, so nothing is compacted between layers (a dropped row is a dead slot).
//   select     before a TopN cut: a windowed histogram of the select keys, summed over the blocks,
//              then the keys of the boundary bin gathered and ranked by every block.
//
// Measured on a B200 (148 blocks): a layer of the 6 x 6 transverse-field Ising quench (threshold
// 1e-5, up to 196,000 terms, f64) took 85 us through the per-layer kernels and takes 14.4 us here;
// a four-word layer with a TopN cut at 50,000 terms 100 us and 21 us.  What bounds it is latency: of
// the 14.4 us the two barriers (with the wait for the slowest block) take 6.4, combining the
// blocks' aggregates 2.2, the merge-path split 1.6, and everything done on the rows 4.2.  512
// threads a block: at a few thousand rows a block more threads only lengthen its own barriers.
//
// The sums, products and comparisons of a layer are those of the per-layer kernels, in the same
// order, so the results are the same bits.  The input store is only read: a run that fails
// leaves it as it was.  A layer that does not fit (rows and partners above what the blocks hold)
// ends the run before it; the rows are then in the work store.
#include <algorithm>
#include <atomic>

#include "ps_device.cuh"
#include "ps_rotlayer.cuh"
#include "ps_run.h"

namespace psb {

namespace {

constexpr uint16_t kDead = 0xFFFF;
constexpr int kWarps = kRunThreads / 32;

// Shared memory of a block, for R rows (R a multiple of 8): keys and coefficients of the rows it
// merged, and per merged slot the row its key comes from (kDead: no row) and its coefficient;
// the partners' slots and divergence ranks.  The partners' offsets and the select's candidates
// take the merged coefficients' place, which only the merge reads.
template <int W, typename T>
struct RunSmem {
    static constexpr size_t row_bytes = 16 * W + sizeof(T) + sizeof(T) + 2 + 2 + 2;
    uint64_t* key;
    T* c;
    T* v;
    uint16_t *src, *plist, *dv;
    int* off;
    uint64_t* cand;
    __device__ RunSmem(unsigned char* p, uint32_t R) {
        key = reinterpret_cast<uint64_t*>(p);
        p += (size_t)R * 16 * W;
        c = reinterpret_cast<T*>(p);
        off = reinterpret_cast<int*>(p);
        cand = reinterpret_cast<uint64_t*>(p);
        p += (size_t)R * sizeof(T);
        v = reinterpret_cast<T*>(p);
        p += (size_t)R * sizeof(T);
        src = reinterpret_cast<uint16_t*>(p);
        p += (size_t)R * 2;
        plist = reinterpret_cast<uint16_t*>(p);
        p += (size_t)R * 2;
        dv = reinterpret_cast<uint16_t*>(p);
    }
};

// Grid barrier on a counter that only grows (zero at launch): every block's writes before it are
// visible after it to loads that bypass L1.  Bounded; false once a wait gave up.
__device__ __forceinline__ bool run_barrier(unsigned int* bar, unsigned int& target, Ctl* ctl, uint32_t info) {
    target += gridDim.x;
    __syncthreads();
    int fail = 0;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(bar, 1u);
        long long spins = 0;
        while ((int)(ld_acquire_u32(bar) - target) < 0) {
            if (++spins > spin_limit(ctl)) {
                raise_err(ctl, ERR_TIMEOUT, info);
                fail = 1;
                break;
            }
        }
        __threadfence();
    }
    return __syncthreads_or(fail) == 0;
}

template <int W>
__device__ __forceinline__ void ldcg_key(const uint64_t* base, uint64_t row, uint64_t (&k)[2 * W]) {
    const ulonglong2* p = reinterpret_cast<const ulonglong2*>(base) + row * W;
#pragma unroll
    for (int q = 0; q < W; ++q) {
        const ulonglong2 x = __ldcg(p + q);
        k[2 * q] = x.x;
        k[2 * q + 1] = x.y;
    }
}

// Warp-wide merge-path split of diagonal d of the rows S[0, n) and P[0, m): (i, j) with i + j = d
// or d + 1, a pair of equal keys (own row, partner) kept together.
template <int W>
__device__ __forceinline__ void run_split(const uint64_t* S, uint64_t n, const uint64_t* P, uint64_t m, uint64_t d,
                                          uint32_t& si, uint32_t& sj) {
    const int lane = threadIdx.x & 31;
    uint64_t lo = d > m ? d - m : 0, hi = d < n ? d : n;
    auto pred = [&](uint64_t i) {  // S[i] <= P[d - 1 - i]
        uint64_t a[2 * W], b[2 * W];
        ldcg_key<W>(S, i, a);
        ldcg_key<W>(P, d - 1 - i, b);
        return le_regs<W>(a, b);
    };
    while (hi - lo > 32) {
        const uint64_t span = hi - lo;
        const unsigned int b = __ballot_sync(0xffffffffu, pred(lo + (span * (uint64_t)lane) / 32));
        const int c = __popc(b);
        if (c == 0) {
            hi = lo;
            break;
        }
        const uint64_t p0 = lo + (span * (uint64_t)(c - 1)) / 32;
        const uint64_t p1 = c < 32 ? lo + (span * (uint64_t)c) / 32 : hi;
        lo = p0 + 1;
        hi = p1;
    }
    const uint64_t span = hi - lo;
    const unsigned int b = __ballot_sync(0xffffffffu, (uint64_t)lane < span ? pred(lo + lane) : false);
    uint64_t i = lo + (uint64_t)__popc(b), j = d - i;
    if (lane == 0) {
        if (i > 0 && j < m) {
            uint64_t a[2 * W], q[2 * W];
            ldcg_key<W>(S, i - 1, a);
            ldcg_key<W>(P, j, q);
            if (eq_regs<W>(a, q)) ++j;
        }
        si = (uint32_t)i;
        sj = (uint32_t)j;
    }
}

// Inclusive sum over the first 256 threads of two counts at once (smem: 2 x kWarps words); every
// thread of the block must call it.
__device__ __forceinline__ void scan_pair(unsigned int& a, unsigned int& b, unsigned int* s) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, b, o);
        if (lane >= o) {
            a += x;
            b += y;
        }
    }
    if (lane == 31) {
        s[warp] = a;
        s[kWarps + warp] = b;
    }
    __syncthreads();
    for (int w = 0; w < warp; ++w) {
        a += s[w];
        b += s[kWarps + w];
    }
}

}  // namespace

template <int W, typename T>
__global__ void __launch_bounds__(kRunThreads, 1) k_layer_run(const RunArgs<W, T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const RunSmem<W, T> S(smem_raw, a.rcap);
    __shared__ RunLayer<W, T> L;
    __shared__ AmpTab<T> A;
    __shared__ NoiseSmem<T> NS;
    __shared__ unsigned int s_drop[kMaxNoise + 1];
    __shared__ unsigned int s_scan[2 * kWarps];
    __shared__ unsigned int s_wa[kWarps], s_wp[kWarps];
    __shared__ uint4 s_fwd[kWarps], s_bwd[kWarps];
    __shared__ unsigned int s_ne[kWarps];
    __shared__ int s_red[kWarps][4 * kRunLevels];
    __shared__ int s_pre[4 * kRunLevels];
    __shared__ unsigned int s_off, s_pbase, s_n, s_m;
    __shared__ uint32_t s_bi[2], s_bj[2];
    __shared__ uint16_t s_si[kRunThreads + 1], s_sj[kRunThreads + 1];
    __shared__ unsigned int s_hist[kRunBins];
    __shared__ unsigned int s_cnt, s_choice, s_above, s_inbin, s_base;
    __shared__ unsigned long long s_boundary;
    static_assert(kRunLevels == 4, "packed scans hold four levels");

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned int lt = (1u << lane) - 1u;
    const unsigned int G = gridDim.x, b = blockIdx.x;
    Ctl* ctl = a.ctl;
    unsigned int target = 0;
    unsigned int epoch = 0, gathers = 0;  // histogram and candidate buffers in turn
    int window = a.window;
    uint64_t wbase = a.window_base, last_boundary = 0;
    int have_boundary = 0;

    // the block's slice of the input
    uint32_t slots;
    {
        const uint64_t r0 = a.n * b / G, r1 = a.n * (b + 1) / G;
        slots = (uint32_t)(r1 - r0);
        const ulonglong2* k2 = reinterpret_cast<const ulonglong2*>(a.Sk) + r0 * W;
        ulonglong2* s2 = reinterpret_cast<ulonglong2*>(S.key);
        for (uint32_t i = tid; i < slots * W; i += kRunThreads) s2[i] = k2[i];
        for (uint32_t i = tid; i < slots; i += kRunThreads) {
            S.v[i] = a.Sc[r0 + i];
            S.src[i] = (uint16_t)i;
        }
    }
    __syncthreads();

    // add `count` (this thread's) to a per-layer counter
    auto count_rows = [&](unsigned int count, unsigned int* to) {
        count = __reduce_add_sync(0xffffffffu, count);
        if (lane == 0 && count) atomicAdd(to, count);
    };

    uint32_t layer = 0;
    for (;; ++layer) {
        const bool done = layer == a.nlayers;
        __syncthreads();  // every thread is done with the last layer's table
        if (!done) {
            const uint32_t* src = reinterpret_cast<const uint32_t*>(a.prog + layer);
            uint32_t* dst = reinterpret_cast<uint32_t*>(&L);
            for (uint32_t i = tid; i < sizeof(RunLayer<W, T>) / 4; i += kRunThreads) dst[i] = __ldg(src + i);
        }
        __syncthreads();
        const int nnoise = done ? 0 : L.noise_n;
        if (!done) {
            if (tid < 16) {
                A.a0[tid] = L.a0[tid];
                A.a1[tid] = L.a1[tid];
            }
            if (nnoise) {
                for (int i = tid; i < nnoise * 4; i += kRunThreads)
                    NS.f[i >> 2][i & 3] = a.noise_f[(size_t)L.noise_first * 4 + i];
                for (int i = tid; i < nnoise; i += kRunThreads) {
                    NS.q[i] = a.noise_q[L.noise_first + i];
                    s_drop[i] = 0;
                }
                if (tid == 0) NS.n = nnoise;
            }
            __syncthreads();
            if (!L.partners) {  // key-preserving: in place, no other block is involved
                unsigned int alive = 0;
                for (uint32_t q = tid; q < slots; q += kRunThreads) {
                    const uint16_t src = S.src[q];
                    if (src == kDead) continue;
                    uint64_t k[2 * W];
                    ld_row<W>(S.key, src, k);
                    const T v = own_coeff<W, T>(L, A, k, S.v[q]);
                    S.v[q] = v;
                    if (v != T(0) && keep_eval<W>(a.keep, k, to_f64(v)))
                        ++alive;
                    else
                        S.src[q] = kDead;
                }
                count_rows(alive, &a.out_rows[layer]);
                count_rows(alive, &a.after_rows[layer]);
                __syncthreads();
                continue;
            }
        }
        // ---- classify: this block's live rows and emitting rows, counted and listed in order
        const uint32_t chunk = ((slots + kWarps - 1) / kWarps + 31) & ~31u;
        const uint32_t c0 = min(slots, warp * chunk), c1 = min(slots, c0 + chunk);
        unsigned int wa = 0, wp = 0;
        for (uint32_t q0 = c0; q0 < c1; q0 += 32) {
            const uint32_t q = q0 + lane;
            const uint16_t src = q < c1 ? S.src[q] : kDead;
            bool e = false;
            if (src != kDead && !done) {
                uint64_t k[2 * W];
                ld_row<W>(S.key, src, k);
                e = emits_partner_regs<W, T>(L, A, k);
            }
            wa += __popc(__ballot_sync(0xffffffffu, src != kDead));
            wp += __popc(__ballot_sync(0xffffffffu, e));
        }
        if (lane == 0) {
            s_wa[warp] = wa;
            s_wp[warp] = wp;
        }
        __syncthreads();
        unsigned int ra = 0, rp = 0, ta = 0, tp = 0;  // ranks before this warp, block totals
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const unsigned int x = s_wa[w], y = s_wp[w];
            ra += w < warp ? x : 0u;
            rp += w < warp ? y : 0u;
            ta += x;
            tp += y;
        }
        if (tp) {
            unsigned int r = rp;
            for (uint32_t q0 = c0; q0 < c1; q0 += 32) {
                const uint32_t q = q0 + lane;
                const uint16_t src = q < c1 ? S.src[q] : kDead;
                bool e = false;
                if (src != kDead) {
                    uint64_t k[2 * W];
                    ld_row<W>(S.key, src, k);
                    e = emits_partner_regs<W, T>(L, A, k);
                }
                const unsigned int be = __ballot_sync(0xffffffffu, e);
                if (e) S.plist[r + __popc(be & lt)] = (uint16_t)q;
                r += __popc(be);
            }
        }
        __syncthreads();
        // ---- divergence ranks and the block's level scans (thread t: partners [pj0, pj1)).  Packed
        // per level: forward (last start + 1) | (last split + 1) << 16, backward first start |
        // first split << 16; the block's first partner counts once the blocks are combined.
        const int NL = done ? 0 : L.nlev;
        const uint32_t jpt = (tp + kRunThreads - 1) / kRunThreads;
        const uint32_t pj0 = min(tp, tid * jpt), pj1 = min(tp, pj0 + jpt);
        unsigned int fwd[4] = {0, 0, 0, 0};
        unsigned int bwd[4] = {~0u, ~0u, ~0u, ~0u};
        if (pj0 < pj1) {
            uint64_t prev[2 * W];
            if (pj0 > 0) ld_row<W>(S.key, S.src[S.plist[pj0 - 1]], prev);
            for (uint32_t j = pj0; j < pj1; ++j) {
                uint64_t k[2 * W];
                ld_row<W>(S.key, S.src[S.plist[j]], k);
                if (j > 0) {
                    const uint32_t d = div_regs<W>(prev, k);
                    S.dv[j] = (uint16_t)d;
#pragma unroll
                    for (int l = 0; l < 4; ++l) {
                        if (l < NL) {
                            const uint32_t rk = L.rank[l];
                            if (d < rk) {
                                fwd[l] = (fwd[l] & 0xFFFF0000u) | (j + 1);
                                if ((bwd[l] & 0xFFFFu) == 0xFFFFu) bwd[l] = (bwd[l] & 0xFFFF0000u) | j;
                            } else if (d == rk) {
                                fwd[l] = (fwd[l] & 0xFFFFu) | ((j + 1) << 16);
                                if ((bwd[l] >> 16) == 0xFFFFu) bwd[l] = (bwd[l] & 0xFFFFu) | (j << 16);
                            }
                        }
                    }
                }
#pragma unroll
                for (int w = 0; w < 2 * W; ++w) prev[w] = k[w];
            }
        }
        if (tp) {  // block-uniform
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                if (l < NL) {
                    unsigned int x = fwd[l], y = bwd[l];
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const unsigned int p = __shfl_up_sync(0xffffffffu, x, o);
                        const unsigned int s = __shfl_down_sync(0xffffffffu, y, o);
                        if (lane >= o) x = __vmaxu2(x, p);
                        if (lane + o < 32) y = __vminu2(y, s);
                    }
                    if (lane == 31) reinterpret_cast<unsigned int*>(&s_fwd[warp])[l] = x;
                    if (lane == 0) reinterpret_cast<unsigned int*>(&s_bwd[warp])[l] = y;
                    const unsigned int ex = __shfl_up_sync(0xffffffffu, x, 1);
                    const unsigned int ey = __shfl_down_sync(0xffffffffu, y, 1);
                    fwd[l] = lane == 0 ? 0u : ex;
                    bwd[l] = lane == 31 ? ~0u : ey;
                }
            }
            __syncthreads();
            unsigned int tf[4] = {0, 0, 0, 0}, tb[4] = {~0u, ~0u, ~0u, ~0u};
            for (int w = 0; w < kWarps; ++w) {
                const uint4 x = s_fwd[w], y = s_bwd[w];
                const unsigned int xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
                for (int l = 0; l < 4; ++l) {
                    if (l < NL) {
                        if (w < warp) fwd[l] = __vmaxu2(fwd[l], xs[l]);
                        if (w > warp) bwd[l] = __vminu2(bwd[l], ys[l]);
                        tf[l] = __vmaxu2(tf[l], xs[l]);
                        tb[l] = __vminu2(tb[l], ys[l]);
                    }
                }
            }
            if (tid == 0) {
                RunSummary<W>& r = a.sums[b];
#pragma unroll
                for (int l = 0; l < 4; ++l) {
                    r.lstart[l] = (uint16_t)((tf[l] & 0xFFFFu) - 1u);
                    r.lsplit[l] = (uint16_t)((tf[l] >> 16) - 1u);
                    r.fstart[l] = (uint16_t)(tb[l] & 0xFFFFu);
                    r.fsplit[l] = (uint16_t)(tb[l] >> 16);
                }
                uint64_t k[2 * W];
                ld_row<W>(S.key, S.src[S.plist[0]], k);
#pragma unroll
                for (int w = 0; w < 2 * W; ++w) r.first[w] = k[w];
                ld_row<W>(S.key, S.src[S.plist[tp - 1]], k);
#pragma unroll
                for (int w = 0; w < 2 * W; ++w) r.last[w] = k[w];
            }
        }
        if (tid == 0) {
            a.sums[b].rows = ta;
            a.sums[b].partners = tp;
        }
        if (!run_barrier(&a.st->bar, target, ctl, 902)) return;
        // ---- place: combine the blocks' aggregates (thread t reads block t's)
        unsigned int rows_t = 0, part_t = 0;
        if (tid < G) {
            rows_t = __ldcg(&a.sums[tid].rows);
            part_t = __ldcg(&a.sums[tid].partners);
        }
        unsigned int rows_in = rows_t, part_in = part_t;
        const unsigned int ne = __ballot_sync(0xffffffffu, part_t > 0);
        if (lane == 0) s_ne[warp] = ne;
        scan_pair(rows_in, part_in, s_scan);  // (its barrier also publishes s_ne)
        const unsigned int pbase_t = part_in - part_t;
        if (tid == b) {
            s_off = rows_in - rows_t;
            s_pbase = pbase_t;
        }
        if (tid == G - 1) {
            s_n = rows_in;
            s_m = part_in;
        }
        if (NL > 0 && tid < ((G + 31) & ~31u)) {  // whole warps
            int fs[4], fp[4], bs[4], bp[4];
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                fs[l] = fp[l] = -1;
                bs[l] = bp[l] = 0x7fffffff;
            }
            if (part_t) {
                // the previous block with partners, whose last key the first key is compared with
                int prev = -1;
                const unsigned int below = ne & lt;
                if (below) {
                    prev = warp * 32 + 31 - __clz(below);
                } else {
                    for (int w = warp - 1; w >= 0; --w)
                        if (s_ne[w]) {
                            prev = w * 32 + 31 - __clz(s_ne[w]);
                            break;
                        }
                }
                const RunSummary<W>& r = a.sums[tid];
                uint32_t d = 0;
                if (prev >= 0) {
                    uint64_t p[2 * W], k[2 * W];
                    ldcg_key<W>(a.sums[prev].last, 0, p);
                    ldcg_key<W>(r.first, 0, k);
                    d = div_regs<W>(p, k);
                }
                const ushort4 ls = __ldcg(reinterpret_cast<const ushort4*>(r.lstart));
                const ushort4 lp = __ldcg(reinterpret_cast<const ushort4*>(r.lsplit));
                const ushort4 gs = __ldcg(reinterpret_cast<const ushort4*>(r.fstart));
                const ushort4 gp = __ldcg(reinterpret_cast<const ushort4*>(r.fsplit));
                const unsigned int lss[4] = {ls.x, ls.y, ls.z, ls.w}, lps[4] = {lp.x, lp.y, lp.z, lp.w};
                const unsigned int gss[4] = {gs.x, gs.y, gs.z, gs.w}, gps[4] = {gp.x, gp.y, gp.z, gp.w};
                const int base = (int)pbase_t;
#pragma unroll
                for (int l = 0; l < 4; ++l) {
                    if (l < NL) {
                        const uint32_t rk = L.rank[l];
                        const bool st = prev < 0 || d < rk, sp = prev >= 0 && d == rk;
                        if ((unsigned int)tid <= b) {  // (the block's own: its first partner only)
                            fs[l] = st ? base : -1;
                            fp[l] = sp ? base : -1;
                            if ((unsigned int)tid < b) {
                                if (lss[l] != 0xFFFFu) fs[l] = base + (int)lss[l];
                                if (lps[l] != 0xFFFFu) fp[l] = base + (int)lps[l];
                            }
                        } else {
                            // (the scans' very first partner starts a group but ends none)
                            bs[l] = st && prev >= 0 ? base : (gss[l] != 0xFFFFu ? base + (int)gss[l] : 0x7fffffff);
                            bp[l] = sp ? base : (gps[l] != 0xFFFFu ? base + (int)gps[l] : 0x7fffffff);
                        }
                    }
                }
            }
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                if (l < NL) {
                    const int x0 = __reduce_max_sync(0xffffffffu, fs[l]), x1 = __reduce_max_sync(0xffffffffu, fp[l]);
                    const int x2 = __reduce_min_sync(0xffffffffu, bs[l]), x3 = __reduce_min_sync(0xffffffffu, bp[l]);
                    if (lane == 0) {
                        s_red[warp][l] = x0;
                        s_red[warp][4 + l] = x1;
                        s_red[warp][8 + l] = x2;
                        s_red[warp][12 + l] = x3;
                    }
                }
            }
        }
        __syncthreads();
        if (tid < 16 && (tid & 3) < NL) {
            int x = s_red[0][tid];
            for (unsigned int w = 1; w < (G + 31) / 32; ++w)
                x = tid < 8 ? max(x, s_red[w][tid]) : min(x, s_red[w][tid]);
            s_pre[tid] = x;
        }
        const uint64_t n = s_n, m = s_m;
        const uint32_t tile = (uint32_t)((n + m + G - 1) / G);
        // every block takes the same decision: the layer fits the blocks and the buffers, or the run ends
        // (a permutation's later steps take at most the same rows again)
        const uint32_t most = !done && L.group > 1 ? (uint32_t)((2 * n + G - 1) / G) : tile;
        const bool fits = most + 1 <= a.rcap && n <= a.wcap && m <= a.pcap;
        // the rows at their positions
        {
            unsigned int r = s_off + ra;
            for (uint32_t q0 = c0; q0 < c1; q0 += 32) {
                const uint32_t q = q0 + lane;
                const uint16_t src = q < c1 ? S.src[q] : kDead;
                const unsigned int bal = __ballot_sync(0xffffffffu, src != kDead);
                if (src != kDead) {
                    const unsigned int pos = r + __popc(bal & lt);
                    if (PS_GUARD(ctl, pos < a.wcap, 903)) {
                        uint64_t k[2 * W];
                        ld_row<W>(S.key, src, k);
                        store_key<W>(a.Wk, pos, k);
                        a.Wc[pos] = S.v[q];
                    }
                }
                r += __popc(bal);
            }
        }
        if (done || !fits) {
            if (b == 0 && tid == 0) {
                a.st->layers_done = layer;
                a.st->n = n;
                a.st->boundary = last_boundary;
                a.st->window = (unsigned int)have_boundary;
            }
            return;
        }
        __syncthreads();  // s_pre
        if (pj0 < pj1) {
            const int base = (int)s_pbase;
            int st[4], sp[4];
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                if (l < NL) {
                    const unsigned int x = fwd[l];
                    st[l] = (x & 0xFFFFu) ? base + (int)(x & 0xFFFFu) - 1 : s_pre[l];
                    sp[l] = (x >> 16) ? base + (int)(x >> 16) - 1 : s_pre[4 + l];
                }
            }
            for (uint32_t j = pj0; j < pj1; ++j) {
                const uint32_t d = j > 0 ? (uint32_t)S.dv[j] : 0xFFFFu;
                int f = 0;
#pragma unroll
                for (int l = 0; l < 4; ++l) {
                    if (l < NL) {
                        const uint32_t rk = L.rank[l];
                        if (d < rk) st[l] = base + (int)j;
                        if (d == rk) sp[l] = base + (int)j;
                        if (sp[l] > st[l]) f -= sp[l] - st[l];
                    }
                }
                S.off[j] = f;
            }
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                if (l < NL) {
                    const unsigned int x = bwd[l];
                    const int e = (x & 0xFFFFu) != 0xFFFFu ? base + (int)(x & 0xFFFFu) : s_pre[8 + l];
                    st[l] = e == 0x7fffffff ? (int)m : e;
                    sp[l] = (x >> 16) != 0xFFFFu ? base + (int)(x >> 16) : s_pre[12 + l];
                }
            }
            for (uint32_t j = pj1; j-- > pj0;) {
                int f = S.off[j];
                const uint32_t d = j > 0 ? (uint32_t)S.dv[j] : 0xFFFFu;
#pragma unroll
                for (int l = 0; l < 4; ++l) {
                    if (l < NL) {
                        if (sp[l] < st[l]) f += st[l] - sp[l];
                        const uint32_t rk = L.rank[l];
                        if (d < rk) st[l] = base + (int)j;
                        if (d == rk) sp[l] = base + (int)j;
                    }
                }
                const long long dest = (long long)base + j + f;
                if (!PS_GUARD(ctl, dest >= 0 && dest < (long long)m, 904)) continue;
                const uint16_t slot = S.plist[j], src = S.src[slot];
                uint64_t k[2 * W];
                ld_row<W>(S.key, src, k);
                T c = S.v[slot];
                const T pc = nnoise && noise_apply<W, T>(NS, a.keep, k, c) < nnoise ? T(0) : partner_coeff<W, T>(L, A, k, c);
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    k[w] ^= L.gx[w];
                    k[W + w] ^= L.gz[w];
                }
                store_key<W>(a.Pk, (uint64_t)dest, k);
                a.Pc[dest] = pc;
            }
        }
        if (!run_barrier(&a.st->bar, target, ctl, 905)) return;
        // ---- merge: this block's share of the merged order
        if (warp < 2) {
            uint64_t d = (uint64_t)(b + warp) * tile;
            if (d > n + m) d = n + m;
            run_split<W>(a.Wk, n, a.Pk, m, d, s_bi[warp], s_bj[warp]);
        }
        __syncthreads();
        const uint32_t i0 = s_bi[0], j0 = s_bj[0], cs = s_bi[1] - i0, cp = s_bj[1] - j0;
        slots = cs + cp;
        {
            // block-uniform; a share that is out of range would be a fault of the split
            const bool ok = s_bi[1] >= i0 && s_bj[1] >= j0 && s_bi[1] <= n && s_bj[1] <= m && slots <= a.rcap;
            if (!PS_GUARD(ctl, ok, 906)) slots = 0;
        }
        const uint32_t cs_ = slots ? cs : 0u;
        {
            const ulonglong2* ks = reinterpret_cast<const ulonglong2*>(a.Wk) + (uint64_t)i0 * W;
            const ulonglong2* kp = reinterpret_cast<const ulonglong2*>(a.Pk) + (uint64_t)j0 * W;
            ulonglong2* s2 = reinterpret_cast<ulonglong2*>(S.key);
            for (uint32_t i = tid; i < slots * W; i += kRunThreads)
                s2[i] = i < cs_ * W ? __ldcg(ks + i) : __ldcg(kp + (i - cs_ * W));
            for (uint32_t i = tid; i < slots; i += kRunThreads) {
                S.c[i] = i < cs_ ? __ldcg(a.Wc + i0 + i) : __ldcg(a.Pc + j0 + (i - cs_));
            }
        }
        __syncthreads();
        const uint32_t cp_ = slots - cs_;
        const uint64_t* sPk = S.key + (size_t)cs_ * 2 * W;
        const uint32_t ipt = (slots + kRunThreads - 1) / kRunThreads;
        {
            const uint32_t dd = min((uint32_t)tid * ipt, slots);
            uint32_t lo = dd > cp_ ? dd - cp_ : 0, hi = min(dd, cs_);
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                uint64_t x[2 * W], y[2 * W];
                ld_row<W>(S.key, mid, x);
                ld_row<W>(sPk, dd - 1 - mid, y);
                if (le_regs<W>(x, y))
                    lo = mid + 1;
                else
                    hi = mid;
            }
            uint32_t i = lo, j = dd - lo;
            if (i > 0 && j < cp_) {
                uint64_t x[2 * W], y[2 * W];
                ld_row<W>(S.key, i - 1, x);
                ld_row<W>(sPk, j, y);
                if (eq_regs<W>(x, y)) ++j;
            }
            s_si[tid] = (uint16_t)i;
            s_sj[tid] = (uint16_t)j;
            if (tid == 0) {
                s_si[kRunThreads] = (uint16_t)cs_;
                s_sj[kRunThreads] = (uint16_t)cp_;
            }
        }
        __syncthreads();
        unsigned int alive = 0;
        const bool inner = L.inner != 0;
        {
            uint32_t i = s_si[tid], j = s_sj[tid];
            const uint32_t ie = s_si[tid + 1], je = s_sj[tid + 1];
            uint64_t x[2 * W], y[2 * W];
            if (i < ie) ld_row<W>(S.key, i, x);
            if (j < je) ld_row<W>(sPk, j, y);
            while (i < ie || j < je) {
                const bool own = (j >= je) || (i < ie && le_regs<W>(x, y));
                const uint32_t q = i + j;
                T v;
                bool ok;
                uint16_t src;
                if (own) {
                    src = (uint16_t)i;
                    T c = S.c[i];
                    int dr = nnoise;
                    if (nnoise) dr = noise_apply<W, T>(NS, a.keep, x, c);
                    if (dr < nnoise) {
                        atomicAdd(&s_drop[dr], 1u);
                        v = T(0);
                    } else {
                        v = own_coeff<W, T>(L, A, x, c);
                    }
                    if (j < je && eq_regs<W>(x, y)) {
                        v = add_rn(v, S.c[cs_ + j]);
                        S.src[q + 1] = kDead;  // the pair's second slot
                        if (++j < je) ld_row<W>(sPk, j, y);
                    }
                    ok = v != T(0) && (inner || keep_eval<W>(a.keep, x, to_f64(v)));
                    if (++i < ie) ld_row<W>(S.key, i, x);
                } else {
                    src = (uint16_t)(cs_ + j);
                    v = S.c[cs_ + j];
                    ok = v != T(0) && (inner || keep_eval<W>(a.keep, y, to_f64(v)));
                    if (++j < je) ld_row<W>(sPk, j, y);
                }
                S.src[q] = ok ? src : kDead;
                S.v[q] = v;
                alive += ok ? 1u : 0u;
            }
        }
        count_rows(alive, &a.out_rows[layer]);
        __syncthreads();
        if (nnoise)
            for (int i = tid; i < nnoise; i += kRunThreads)
                if (s_drop[i]) atomicAdd(&a.drops[L.noise_first + i], s_drop[i]);
        if (a.topn == 0 || n + m <= a.topn || L.wide == 2) {  // (a permutation adds no row)
            if (a.topn) count_rows(alive, &a.after_rows[layer]);
            continue;
        }
        // ---- select: the boundary among the live rows' select keys.  kk = key - lowkey (the window's
        // base, or 0), known so far: kk >> shift == prefix, `rank` left among those `inbin` rows.
        bool full = !window, keep_all = false;
        uint64_t lowkey = 0, prefix = 0;
        unsigned int rank = 0, inbin = 0;
        int shift = 0;
        bool first_digit = true;
        for (;;) {
            for (int i = tid; i < kRunBins; i += kRunThreads) s_hist[i] = 0;
            __syncthreads();
            int bits;
            if (first_digit) {
                lowkey = full ? 0ull : wbase;
                shift = full ? 52 : 44;  // octaves of |c|^2, or 1/256 octaves around the last boundary
                bits = 11;
            } else {
                bits = min(11, shift);
                shift -= bits;
            }
            for (uint32_t q = tid; q < slots; q += kRunThreads) {
                const uint16_t src = S.src[q];
                if (src == kDead) continue;
                const uint64_t mk = mag_key<T>(S.v[q]);
                if (first_digit) {
                    const uint64_t bin = mk < lowkey ? 0ull : (mk - lowkey) >> shift;
                    atomicAdd(&s_hist[bin > 2047 ? 2047u : (unsigned int)bin], 1u);
                } else if (mk >= lowkey && ((mk - lowkey) >> (shift + bits)) == prefix) {
                    atomicAdd(&s_hist[(unsigned int)((mk - lowkey) >> shift) & ((1u << bits) - 1u)], 1u);
                }
            }
            __syncthreads();
            unsigned int* hist = a.st->hist[epoch % 3];
            for (int i = tid; i < kRunBins; i += kRunThreads)
                if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
            if (!run_barrier(&a.st->bar, target, ctl, 907)) return;
            {
                // thread t holds bins 2047 - 4 t - {0..3}, counted from the top
                const uint4 h4 = __ldcg(reinterpret_cast<const uint4*>(hist) + (kRunThreads - 1 - tid));
                const unsigned int c4[4] = {h4.w, h4.z, h4.y, h4.x};
                unsigned int incl = c4[0] + c4[1] + c4[2] + c4[3], zero = 0;
                const unsigned int mine = incl;
                scan_pair(incl, zero, s_scan);
                if (tid == kRunThreads - 1) s_cnt = incl;
                if (tid == 0) {
                    s_choice = 0;
                    s_above = 0;
                    s_inbin = 0;
                }
                __syncthreads();
                const unsigned int want = first_digit ? (unsigned int)a.topn : rank;
                unsigned int acc = incl - mine;
                if (acc < want && incl >= want) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (acc + c4[i] >= want) {
                            s_choice = (unsigned int)(kRunBins - 1 - 4 * tid - i);
                            s_above = acc;
                            s_inbin = c4[i];
                            break;
                        }
                        acc += c4[i];
                    }
                }
                // the buffer of the round before last: every block has read it, and it is used after
                // the next round's barrier
                unsigned int* old = a.st->hist[(epoch + 2) % 3];
                for (unsigned int i = b * kRunThreads + tid; i < (unsigned int)kRunBins; i += G * kRunThreads) old[i] = 0;
                ++epoch;
            }
            __syncthreads();
            if (first_digit) {
                if (s_cnt <= a.topn) {
                    keep_all = true;
                    break;
                }
                if (!full && (s_choice == 0 || s_choice == 2047)) {
                    full = true;  // the boundary left the window
                    continue;
                }
                prefix = s_choice;
                rank = (unsigned int)a.topn - s_above;
                first_digit = false;
            } else {
                prefix = prefix << bits | s_choice;
                rank -= s_above;
            }
            inbin = s_inbin;
            if (inbin <= (unsigned int)kRunCand || shift == 0) break;
        }
        if (!keep_all) {
            unsigned int ties = inbin;
            uint64_t boundary;
            if (shift == 0) {
                boundary = prefix + lowkey;
            } else {
                // the bin's keys, gathered from every block and ranked by every block
                __syncthreads();
                if (tid == 0) s_cnt = 0;
                __syncthreads();
                for (uint32_t q = tid; q < slots; q += kRunThreads) {
                    const uint16_t src = S.src[q];
                    if (src == kDead) continue;
                    const uint64_t mk = mag_key<T>(S.v[q]);
                    if (mk >= lowkey && ((mk - lowkey) >> shift) == prefix) {
                        const unsigned int at = atomicAdd(&s_cnt, 1u);
                        if (PS_GUARD(ctl, at < (unsigned int)kRunCand, 908)) S.cand[at] = mk;
                    }
                }
                __syncthreads();
                const unsigned int have = min(s_cnt, (unsigned int)kRunCand);
                if (tid == 0) s_base = have ? atomicAdd(&a.st->cand_n[gathers % 3], have) : 0u;
                __syncthreads();
                unsigned long long* list = a.st->cand[gathers & 1];
                for (unsigned int i = tid; i < have; i += kRunThreads)
                    if (PS_GUARD(ctl, s_base + i < (unsigned int)kRunCand, 909)) list[s_base + i] = S.cand[i];
                if (!run_barrier(&a.st->bar, target, ctl, 910)) return;
                for (unsigned int i = tid; i < inbin; i += kRunThreads) S.cand[i] = __ldcg(&list[i]);
                if (b == 0 && tid == 0) a.st->cand_n[(gathers + 2) % 3] = 0;
                ++gathers;
                __syncthreads();
                for (unsigned int i = tid; i < inbin; i += kRunThreads) {
                    const uint64_t mine = S.cand[i];
                    unsigned int above = 0, same = 0;
                    for (unsigned int q = 0; q < inbin; ++q) {
                        const uint64_t o = S.cand[q];
                        above += o > mine ? 1u : 0u;
                        same += o == mine ? 1u : 0u;
                    }
                    if (above < rank && rank <= above + same) {  // (every holder of the boundary agrees)
                        s_boundary = mine;
                        s_above = above;
                        s_inbin = same;
                    }
                }
                __syncthreads();
                boundary = s_boundary;
                rank -= s_above;
                ties = s_inbin;
            }
            last_boundary = boundary;
            have_boundary = boundary != 0;
            window = boundary != 0;
            wbase = boundary > (1024ull << 44) ? boundary - (1024ull << 44) : 0ull;
            // rows above the boundary stay; of the rows equal to it the first `rank` in key order
            // (none when it is NaN's key)
            unsigned int before = 0;  // ties in the blocks before this one, when the quota cuts them
            const bool cut = boundary != 0 && rank < ties;
            if (cut) {
                unsigned int t = 0;
                for (uint32_t q = tid; q < slots; q += kRunThreads) {
                    const uint16_t src = S.src[q];
                    t += src != kDead && mag_key<T>(S.v[q]) == boundary ? 1u : 0u;
                }
                __syncthreads();
                if (tid == 0) s_cnt = 0;
                __syncthreads();
                count_rows(t, &s_cnt);
                __syncthreads();
                if (tid == 0) a.st->ties[b] = s_cnt;
                if (!run_barrier(&a.st->bar, target, ctl, 911)) return;
                unsigned int x = (unsigned int)tid < b ? __ldcg(&a.st->ties[tid]) : 0u, zero = 0;
                scan_pair(x, zero, s_scan);
                if (tid == kRunThreads - 1) s_base = x;
                __syncthreads();
                before = s_base;
            }
            const uint32_t ch = ((slots + kWarps - 1) / kWarps + 31) & ~31u;
            const uint32_t w0 = min(slots, warp * ch), w1 = min(slots, w0 + ch);
            unsigned int wt = 0;
            if (cut) {
                for (uint32_t q0 = w0; q0 < w1; q0 += 32) {
                    const uint32_t q = q0 + lane;
                    const uint16_t src = q < w1 ? S.src[q] : kDead;
                    wt += __popc(__ballot_sync(0xffffffffu, src != kDead && mag_key<T>(S.v[q]) == boundary));
                }
                if (lane == 0) s_wa[warp] = wt;
                __syncthreads();
                wt = before;
                for (int w = 0; w < warp; ++w) wt += s_wa[w];
            }
            alive = 0;
            for (uint32_t q0 = w0; q0 < w1; q0 += 32) {
                const uint32_t q = q0 + lane;
                const uint16_t src = q < w1 ? S.src[q] : kDead;
                const uint64_t mk = src != kDead ? mag_key<T>(S.v[q]) : 0ull;
                const bool tie = src != kDead && mk == boundary && boundary != 0;
                bool keep = src != kDead && (mk > boundary || tie);
                if (cut) {
                    const unsigned int bt = __ballot_sync(0xffffffffu, tie);
                    if (tie && wt + __popc(bt & lt) >= rank) keep = false;
                    wt += __popc(bt);
                }
                if (src != kDead && !keep) S.src[q] = kDead;
                alive += keep ? 1u : 0u;
            }
        }
        count_rows(alive, &a.after_rows[layer]);
        __syncthreads();
    }
}

template <int W, typename T>
uint32_t RunOps<W, T>::rows_per_block() {
    static std::atomic<int> cache{0};
    int v = cache.load(std::memory_order_relaxed);
    if (v == 0) {
        const void* kern = (const void*)k_layer_run<W, T>;
        int dev = 0, coop = 0, optin = 0, per = 0;
        cudaFuncAttributes at;
        v = -1;
        if (cudaGetDevice(&dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop &&
            cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess &&
            cudaFuncGetAttributes(&at, kern) == cudaSuccess) {
            constexpr size_t row = RunSmem<W, T>::row_bytes;
            const size_t rows = ((size_t)optin - at.sharedSizeBytes) / row / 8 * 8;
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(rows * row)) == cudaSuccess &&
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, kRunThreads, rows * row) == cudaSuccess && per > 0)
                v = (int)std::min<size_t>(rows, 65528);  // (16-bit slots)
        }
        cudaGetLastError();
        cache.store(v, std::memory_order_relaxed);
    }
    return v > 0 ? (uint32_t)v : 0u;
}

template <int W, typename T>
cudaError_t RunOps<W, T>::launch(const RunArgs<W, T>& a, int blocks, cudaStream_t st, KernelProf* prof) {
    if (a.rcap == 0 || a.rcap > rows_per_block()) return cudaErrorNotSupported;
    void* args[] = {(void*)&a};
    prof->begin(K_LAYER_RUN, 0.0, st);
    const cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_layer_run<W, T>, dim3((unsigned)blocks),
                                                      dim3(kRunThreads), args, RunSmem<W, T>::row_bytes * a.rcap, st);
    prof->end(st);
    return e;
}

template struct RunOps<1, double>;
template struct RunOps<1, float>;
template struct RunOps<2, double>;
template struct RunOps<2, float>;
template struct RunOps<4, double>;
template struct RunOps<4, float>;

}  // namespace psb
