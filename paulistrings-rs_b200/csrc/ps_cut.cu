// ps_cut.cu -- TopN between rotation layers without a compaction.
//
// At a TopN budget a layer's merge leaves a few percent more rows than the budget, and compacting
// them moved the whole sum once more only to drop those.  Instead the rows stay in the merge's
// slots: the cut finds the boundary, and a row is live iff its select key reaches it.  The next
// layer reads the slots in place (k_merge's CUT form drops the dead rows as it reads them), so a
// layer reads and writes the sum once.
//
//   k_topn_cut    one pass over the coefficients and the merge's partner-test bytes, each block a
//                 run of tiles in order: the window's boundary bin is known from the merge's
//                 histogram, its keys go to the block's candidate list; per tile the rows that emit
//                 a partner under the next layer are listed with their divergence ranks, and the
//                 level scans' aggregates (ps_rotation.cu) are combined along the run.  The last
//                 block to finish combines the blocks and selects the boundary among the candidates.
//   k_cut_place   a warp per tile: both level scans finished for its listed rows, each partner
//                 written at its sorted slot; a dead row's partner is a zero, which adds nothing to an
//                 equal row and is dropped otherwise.
//   k_cut_partition  merge-path split points over the slots (the row index goes through pr).
//
// Measured on a B200 (random two-qubit rotation layers, 64 qubits, f64, TopN 2^25; us a layer): the
// compaction 404, select 168, level scans 56 and placement 119 they replace became the cut's 234 and
// the placement's 140, and the merge, which reads the dropped rows once more and its own coefficients
// row by row from the slots, went from 477 to 637; a layer from 1276 to 1061.  At 10^6 terms (8 x 8
// quench) a layer went from 193 to 125 us: fewer launches and no look-back.  The cut reads 8 bytes a
// row and gathers the listed keys, 64 bytes of DRAM each for 16: about 3 TB/s at that size.  At 10^6
// terms it is latency: 25 us for its tiles (three warps of a block have one each), 8 along the run,
// 15 in the last block.  Placing from rows the cut stored side by side instead of gathering them
// again: 222 against 242 us, but the cut 463 against 409 (2^26); not kept.
//
// No kernel here waits for another block.  A pass the cut cannot serve (the boundary left the
// window, more equal magnitudes at the boundary than the lists hold) reports it and changes nothing;
// the caller selects and compacts as before.
#include <algorithm>

#include "ps_cut.h"
#include "ps_device.cuh"
#include "ps_rotlayer.cuh"
#include "ps_store.h"

namespace psb {

namespace {

constexpr int kCutWarps = kCutThreads / 32;
constexpr int kPlaceThreads = 256;
constexpr int kCutRows = 1288;  // rows of a tile's slot, at most
constexpr size_t kCutListBytes = (size_t)kCutWarps * kCutRows * 2;
constexpr size_t kCutSmem = kCutListBytes + (size_t)kCutBlockCand * 12;
static_assert(kCutListBytes >= 2048 * 4 && kCutListBytes % 16 == 0, "the histogram takes the lists' place");
constexpr int kNV = 2 * kCutLevels;  // starts, then splits

// Exclusive block scan (kCutThreads threads) of v by op with identity id; s: kCutWarps words.
// `total` is the reduction over the block.  Ends with a barrier.
template <bool kSuffix, typename Op>
__device__ __forceinline__ int cut_scan(int v, int id, int* s, int& total, Op op) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = kSuffix ? __shfl_down_sync(0xffffffffu, x, o) : __shfl_up_sync(0xffffffffu, x, o);
        if (kSuffix ? lane + o < 32 : lane >= o) x = op(x, y);
    }
    if (lane == (kSuffix ? 0 : 31)) s[warp] = x;
    const int e = kSuffix ? __shfl_down_sync(0xffffffffu, x, 1) : __shfl_up_sync(0xffffffffu, x, 1);
    int r = lane == (kSuffix ? 31 : 0) ? id : e;
    __syncthreads();
    int t = id;
#pragma unroll
    for (int w = 0; w < kCutWarps; ++w) {
        const int y = s[w];
        if (kSuffix ? w > warp : w < warp) r = op(r, y);
        t = op(t, y);
    }
    total = t;
    __syncthreads();
    return r;
}
struct OpAdd {
    __device__ int operator()(int a, int b) const { return a + b; }
};
struct OpMax {
    __device__ int operator()(int a, int b) const { return max(a, b); }
};
struct OpMin {
    __device__ int operator()(int a, int b) const { return min(a, b); }
};

}  // namespace

template <int W, typename T>
__global__ void __launch_bounds__(kCutThreads, W == 4 ? 1 : 2) k_topn_cut(const CutArgs<W, T> a) {
    Ctl* ctl = a.ctl;
    if (ctl->err) return;  // the layer failed: its caller restores the store
    // lists of the warps' tiles (reused as the last block's histogram) and the block's candidates
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint16_t* lst = reinterpret_cast<uint16_t*>(smem_raw) + (threadIdx.x >> 5) * kCutRows;
    unsigned int* s_hist = reinterpret_cast<unsigned int*>(smem_raw);
    uint64_t* s_ckey = reinterpret_cast<uint64_t*>(smem_raw + kCutListBytes);
    uint32_t* s_crow = reinterpret_cast<uint32_t*>(smem_raw + kCutListBytes + kCutBlockCand * 8);
    __shared__ int s_scan[kCutWarps];
    __shared__ unsigned int s_choice, s_above, s_inbin, s_cand, s_base, s_last, s_tie;
    __shared__ int s_first_tile;
    __shared__ unsigned long long s_bound;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t G = gridDim.x, b = blockIdx.x, SR = a.slot_rows;
    const uint32_t ntiles = (uint32_t)(ctl->span / SR);
    const uint32_t tpb = (ntiles + G - 1) / G;
    const uint32_t t0 = min(ntiles, b * tpb), t1 = min(ntiles, t0 + tpb);
    const int NL = a.next.n;

    // the boundary bin, from the merge's window histogram (every block the same)
    bool missed;
    unsigned int choice, above;
    {
        const uint4 h4 = reinterpret_cast<const uint4*>(a.hist)[kCutThreads - 1 - tid];
        const unsigned int c4[4] = {h4.w, h4.z, h4.y, h4.x};
        const int mine = (int)(c4[0] + c4[1] + c4[2] + c4[3]);
        if (tid == 0) s_choice = s_above = s_inbin = s_cand = 0;
        int total;
        unsigned int acc = (unsigned int)cut_scan<false>(mine, 0, s_scan, total, OpAdd());
        const unsigned int want = (unsigned int)a.keep_n;
        if (acc < want && acc + (unsigned int)mine >= want) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (acc + c4[i] >= want) {
                    s_choice = (unsigned int)(2047 - 4 * tid - i);
                    s_above = acc;
                    s_inbin = c4[i];
                    break;
                }
                acc += c4[i];
            }
        }
        __syncthreads();
        const bool keep_all = (unsigned long long)(unsigned int)total <= a.keep_n;
        choice = s_choice;
        above = s_above;
        // (a sum within its budget has no boundary to cut at: the caller compacts it)
        missed = keep_all || choice == 0 || choice == 2047 || s_inbin > kCutCand;
    }
    const bool collect = !missed;
    int low_bits;
    const uint64_t low = cut_bin_low(choice, a.base, low_bits);
    // the bin as a range of |c|^2
    const double q_low = __longlong_as_double((long long)low),
                 q_high = __longlong_as_double((long long)(low + (1ull << low_bits)));

    // ---- this block's tiles, a warp per tile
    for (uint32_t t = t0 + warp; t < t1; t += kCutWarps) {
        const uint32_t cnt = min(__ldg(a.count + t), SR);
        const uint64_t row0 = (uint64_t)t * SR;
        // the boundary bin's rows: eight groups' loads in flight
        if (collect) {
            constexpr int U = 8;
            for (uint32_t r0 = 0; r0 < cnt; r0 += 32 * U) {
                T c[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t r = r0 + 32 * u + lane;
                    c[u] = r < cnt ? a.coef[row0 + r] : T(0);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const double q = __dmul_rn(to_f64(c[u]), to_f64(c[u]));
                    if (q >= q_low && q < q_high) {  // (q_low > 0: no row past the tile's last)
                        const uint64_t mk = (uint64_t)__double_as_longlong(q);
                        const uint32_t row = (uint32_t)(row0 + r0 + 32 * u + lane);
                        const unsigned int at = atomicAdd(&s_cand, 1u);
                        if (at < kCutBlockCand) {
                            s_ckey[at] = mk;
                            s_crow[at] = row;
                        } else {  // (a wide bin at a large sum)
                            const unsigned int g = atomicAdd(&a.state->ncand, 1u);
                            if (g < kCutCand) {
                                a.cand[g] = mk;
                                a.cand_row[g] = row;
                            }
                        }
                    }
                }
            }
        }
        // the rows that emit a partner, in order, from the merge's bytes (16 a lane)
        unsigned int pc = 0;
        const uint32_t words = (cnt + 15) / 16;
        const uint4* fl = reinterpret_cast<const uint4*>(a.flags + (uint64_t)t * flag_stride(SR));
        for (uint32_t w0 = 0; w0 < words; w0 += 32) {
            const uint32_t w = w0 + lane;
            unsigned int bits = 0;
            if (w < words) {
                const uint4 x = fl[w];
                // four 0 / 1 bytes to four bits, the first byte lowest
                auto pack = [](unsigned int y) { return ((y & 0x01010101u) * 0x01020408u) >> 24; };
                bits = pack(x.x) | pack(x.y) << 4 | pack(x.z) << 8 | pack(x.w) << 12;
                if (w == words - 1 && (cnt & 15)) bits &= (1u << (cnt & 15)) - 1u;  // past the tile's rows: stale
            }
            const unsigned int mine = __popc(bits);
            unsigned int incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            unsigned int at = pc + incl - mine;
            while (bits) {
                lst[at++] = (uint16_t)(w * 16 + (__ffs(bits) - 1));
                bits &= bits - 1;
            }
            pc += __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncwarp();
        // the listed rows: ranks from the one before, and per level the last and first start and split
        int ls[kNV], fs[kNV];
#pragma unroll
        for (int l = 0; l < kNV; ++l) {
            ls[l] = -1;
            fs[l] = kCutNone;
        }
        uint64_t prev[2 * W];
#pragma unroll
        for (int w = 0; w < 2 * W; ++w) prev[w] = 0;
        constexpr int V = W == 1 ? 4 : (W == 2 ? 2 : 1);
        for (uint32_t j0 = 0; j0 < pc; j0 += 32 * V) {
            uint64_t k[V][2 * W];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const uint32_t j = j0 + 32 * v + lane;
#pragma unroll
                for (int w = 0; w < 2 * W; ++w) k[v][w] = 0;
                if (j < pc) load_key<W>(a.keys, row0 + lst[j], k[v]);
            }
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const uint32_t j = j0 + 32 * v + lane;
                uint64_t pk[2 * W];
#pragma unroll
                for (int w = 0; w < 2 * W; ++w) {
                    const uint64_t up = __shfl_up_sync(0xffffffffu, k[v][w], 1);
                    pk[w] = lane == 0 ? prev[w] : up;
                    prev[w] = __shfl_sync(0xffffffffu, k[v][w], 31);  // (used only when the group is full)
                }
                uint32_t d = kDivUnknown;
                if (j < pc) {
                    if (j > 0) d = div_regs<W>(pk, k[v]);
                    a.plist[row0 + j] = lst[j];
                    a.D[row0 + j] = (uint16_t)d;
                }
#pragma unroll
                for (int q = 0; q < kCutLevels; ++q) {
                    if (q < NL) {
                        const uint32_t rk = a.next.rank[q];
                        const unsigned int bs = __ballot_sync(0xffffffffu, d < rk);
                        const unsigned int bp = __ballot_sync(0xffffffffu, d == rk);
                        const int at = (int)(j0 + 32 * v);
                        if (bs) {
                            ls[q] = at + 31 - __clz(bs);
                            if (fs[q] == kCutNone) fs[q] = at + __ffs(bs) - 1;
                        }
                        if (bp) {
                            ls[kCutLevels + q] = at + 31 - __clz(bp);
                            if (fs[kCutLevels + q] == kCutNone) fs[kCutLevels + q] = at + __ffs(bp) - 1;
                        }
                    }
                }
            }
        }
        __syncwarp();
        if (lane == 0) {
            CutTile& o = a.tiles[t];
            o.partners = pc;
#pragma unroll
            for (int l = 0; l < kNV; ++l) {
                o.fwd[l] = ls[l];
                o.bwd[l] = fs[l];
            }
        }
    }
    __syncthreads();
    const unsigned int mine_c = min(s_cand, kCutBlockCand);
    if (tid == 0) {
        s_base = mine_c ? atomicAdd(&a.state->ncand, mine_c) : 0u;
        s_first_tile = -1;
    }
    __syncthreads();
    for (unsigned int i = tid; i < mine_c; i += kCutThreads) {
        if (s_base + i < kCutCand) {
            a.cand[s_base + i] = s_ckey[i];
            a.cand_row[s_base + i] = s_crow[i];
        }
    }
    // ---- along the run: rows and partners before each tile, ranks across tiles, scans' prefixes
    int rows_run = 0, part_run = 0, ne_run = -1, fwd_run[kNV], bwd_run[kNV];
#pragma unroll
    for (int l = 0; l < kNV; ++l) {
        fwd_run[l] = -1;
        bwd_run[l] = kCutNone;
    }
    for (uint32_t q0 = t0; q0 < t1; q0 += kCutThreads) {
        const uint32_t t = q0 + tid;
        const bool have = t < t1;
        const int rows = have ? (int)min(__ldg(a.count + t), SR) : 0;
        const int parts = have ? (int)a.tiles[t].partners : 0;
        int tot;
        const int rb = rows_run + cut_scan<false>(rows, 0, s_scan, tot, OpAdd());
        rows_run += tot;
        const int pb = part_run + cut_scan<false>(parts, 0, s_scan, tot, OpAdd());
        part_run += tot;
        const int pne = max(ne_run, cut_scan<false>(parts ? (int)t : -1, -1, s_scan, tot, OpMax()));
        ne_run = max(ne_run, tot);
        uint32_t d = kDivUnknown;
        if (parts) {
            const uint64_t at = (uint64_t)t * SR;
            if (pne >= 0) {
                const uint64_t pat = (uint64_t)pne * SR;
                uint64_t p[2 * W], k[2 * W];
                load_key<W>(a.keys, pat + a.plist[pat + a.tiles[pne].partners - 1], p);
                load_key<W>(a.keys, at + a.plist[at], k);
                d = div_regs<W>(p, k);
                a.D[at] = (uint16_t)d;
            } else {
                s_first_tile = (int)t;  // one thread of one round
            }
        }
        uint32_t flags = 0;
        int ct[kNV], pre[kNV];
#pragma unroll
        for (int l = 0; l < kNV; ++l) ct[l] = -1;
        if (parts) {
            for (int l = 0; l < NL; ++l) flags |= (d < a.next.rank[l] ? 1u : 0u) << l | (d == a.next.rank[l] ? 16u : 0u) << l;
#pragma unroll
            for (int l = 0; l < kNV; ++l) {
                const int x = a.tiles[t].fwd[l];
                ct[l] = x >= 0 ? pb + x : ((flags >> l) & 1u ? pb : -1);
            }
        }
#pragma unroll
        for (int l = 0; l < kNV; ++l) {
            if ((l & (kCutLevels - 1)) < NL) {
                pre[l] = max(fwd_run[l], cut_scan<false>(ct[l], -1, s_scan, tot, OpMax()));
                fwd_run[l] = max(fwd_run[l], tot);
                if ((flags >> l) & 1u) pre[l] = pb;
            } else {
                pre[l] = -1;
            }
        }
        if (have) {
            CutTile& o = a.tiles[t];
            o.rows_before = (uint32_t)rb;
            o.part_before = (uint32_t)pb;
            o.flags = flags;
#pragma unroll
            for (int l = 0; l < kNV; ++l) o.fwd[l] = pre[l];
        }
    }
    const uint32_t rounds = (t1 - t0 + kCutThreads - 1) / kCutThreads;
    for (uint32_t q = 0; q < rounds; ++q) {  // backwards: thread order is tile order within a round
        const uint32_t q0 = t0 + (rounds - 1 - q) * kCutThreads;
        const uint32_t t = q0 + tid;
        const bool have = t < t1;
        int tot;
        CutTile* o = a.tiles + (have ? t : t0);
        const int parts = have ? (int)o->partners : 0;
        const int pb = have ? (int)o->part_before : 0;
        const uint32_t flags = have ? o->flags : 0u;
#pragma unroll
        for (int l = 0; l < kNV; ++l) {
            if ((l & (kCutLevels - 1)) < NL) {
                int ct = kCutNone;
                if (parts) {
                    const int x = o->bwd[l];
                    ct = (flags >> l) & 1u ? pb : (x != kCutNone ? pb + x : kCutNone);
                }
                const int suf = min(bwd_run[l], cut_scan<true>(ct, kCutNone, s_scan, tot, OpMin()));
                bwd_run[l] = min(bwd_run[l], tot);
                if (have) o->bwd[l] = suf;
            }
        }
    }
    if (tid == 0) {
        CutBlock& o = a.blocks[b];
        o.rows = (uint32_t)rows_run;
        o.partners = (uint32_t)part_run;
        o.first_tile = s_first_tile < 0 ? 0u : (uint32_t)s_first_tile;
        if (part_run) {
            const uint64_t f = (uint64_t)s_first_tile * SR, e = (uint64_t)ne_run * SR;
            o.first_row = (uint32_t)(f + a.plist[f]);
            o.last_row = (uint32_t)(e + a.plist[e + a.tiles[ne_run].partners - 1]);
        }
#pragma unroll
        for (int l = 0; l < kNV; ++l) {
            o.fwd[l] = fwd_run[l];
            o.bwd[l] = bwd_run[l];
        }
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        s_last = atomicAdd(&a.state->ticket, 1u) == G - 1 ? 1u : 0u;
        __threadfence();
    }
    __syncthreads();
    if (!s_last) return;

    // ---- the last block: the blocks' places (thread t: block t; G <= kCutThreads)
    {
        const bool have = tid < (int)G;
        CutBlock* o = a.blocks + (have ? tid : 0);
        const int rows = have ? (int)__ldcg(&o->rows) : 0, parts = have ? (int)__ldcg(&o->partners) : 0;
        int tot_rows, tot_parts, tot;
        const int rb = cut_scan<false>(rows, 0, s_scan, tot_rows, OpAdd());
        const int pb = cut_scan<false>(parts, 0, s_scan, tot_parts, OpAdd());
        const int pne = cut_scan<false>(parts ? tid : -1, -1, s_scan, tot, OpMax());
        uint32_t d = kDivStart;
        if (parts) {
            if (pne >= 0) {
                uint64_t p[2 * W], k[2 * W];
                load_key<W>(a.keys, __ldcg(&a.blocks[pne].last_row), p);
                load_key<W>(a.keys, __ldcg(&o->first_row), k);
                d = div_regs<W>(p, k);
            }
            a.D[(uint64_t)__ldcg(&o->first_tile) * SR] = (uint16_t)d;
        }
        int pre[kNV], suf[kNV];
#pragma unroll
        for (int l = 0; l < kNV; ++l) {
            pre[l] = -1;
            suf[l] = kCutNone;
            const int lv = l & (kCutLevels - 1);
            if (lv < NL) {
                const uint32_t rk = a.next.rank[lv];
                // the scans' very first partner starts every group and ends none
                const bool first = parts && (l < kCutLevels ? (pne < 0 || d < rk) : (pne >= 0 && d == rk));
                int ct = -1, cb = kCutNone;
                if (parts) {
                    const int x = __ldcg(&o->fwd[l]), y = __ldcg(&o->bwd[l]);
                    ct = x >= 0 ? pb + x : (first ? pb : -1);
                    cb = first && pne >= 0 ? pb : (y != kCutNone ? pb + y : kCutNone);
                }
                pre[l] = cut_scan<false>(ct, -1, s_scan, tot, OpMax());
                if (first) pre[l] = pb;
                suf[l] = cut_scan<true>(cb, kCutNone, s_scan, tot, OpMin());
            }
        }
        if (have) {
#pragma unroll
            for (int l = 0; l < kNV; ++l) {
                o->fwd[l] = pre[l];
                o->bwd[l] = suf[l];
            }
            o->rbase = (uint32_t)rb;
            o->pbase = (uint32_t)pb;
        }
        if (tid == 0) {
            a.state->rows = (unsigned long long)(unsigned int)tot_rows;
            a.state->partners = (unsigned long long)(unsigned int)tot_parts;
            ctl->count[0] = (unsigned long long)(unsigned int)tot_parts;
        }
    }
    for (int i = tid; i < 2048; i += kCutThreads) a.hist[i] = 0;  // every block has read it
    // ---- the boundary among the candidates: 11-bit digits of the bin's low bits until at most
    // kCutBlockCand keys are left, which are ranked among themselves
    unsigned long long boundary = 0, nabove = 0;
    unsigned int status = missed ? 1u : 0u, last_tie = kCutAllTies;
    if (collect) {
        const unsigned int total = __ldcg(&a.state->ncand);
        unsigned int rank = (unsigned int)a.keep_n - above, inbin = s_inbin;
        uint64_t prefix = 0;  // of pattern - low
        int shift = low_bits;
        if (total != inbin) status = 1u;  // (the merge's count)
        constexpr int U = 4;
        while (status == 0 && inbin > kCutBlockCand && shift > 0) {  // block-uniform
            const int bits = min(11, shift), up = shift;
            shift -= bits;
            for (int i = tid; i < 2048; i += kCutThreads) s_hist[i] = 0;
            __syncthreads();
            for (unsigned int i0 = 0; i0 < total; i0 += kCutThreads * U) {
                uint64_t kk[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const unsigned int i = i0 + u * kCutThreads + tid;
                    kk[u] = i < total ? __ldcg(reinterpret_cast<const unsigned long long*>(a.cand) + i) - low : ~0ull;
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if ((kk[u] >> up) == prefix) atomicAdd(&s_hist[(unsigned int)(kk[u] >> shift) & ((1u << bits) - 1u)], 1u);
            }
            __syncthreads();
            const unsigned int c4[4] = {s_hist[2047 - 4 * tid], s_hist[2046 - 4 * tid], s_hist[2045 - 4 * tid],
                                        s_hist[2044 - 4 * tid]};
            const int mine = (int)(c4[0] + c4[1] + c4[2] + c4[3]);
            int tot;
            unsigned int acc = (unsigned int)cut_scan<false>(mine, 0, s_scan, tot, OpAdd());
            if (acc < rank && acc + (unsigned int)mine >= rank) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (acc + c4[i] >= rank) {
                        s_choice = (unsigned int)(2047 - 4 * tid - i);
                        s_above = acc;
                        s_inbin = c4[i];
                        break;
                    }
                    acc += c4[i];
                }
            }
            __syncthreads();
            prefix = prefix << bits | s_choice;
            rank -= s_above;
            inbin = s_inbin;
            __syncthreads();
        }
        if (inbin > kCutBlockCand) status = 1u;  // that many equal keys
        if (status == 0) {
            if (tid == 0) s_cand = 0;
            __syncthreads();
            for (unsigned int i0 = 0; i0 < total; i0 += kCutThreads * U) {
                uint64_t mk[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const unsigned int i = i0 + u * kCutThreads + tid;
                    mk[u] = i < total ? __ldcg(reinterpret_cast<const unsigned long long*>(a.cand) + i) : 0ull;
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const unsigned int i = i0 + u * kCutThreads + tid;
                    if (i < total && ((mk[u] - low) >> shift) == prefix) {
                        const unsigned int at = atomicAdd(&s_cand, 1u);
                        if (at < kCutBlockCand) {
                            s_ckey[at] = mk[u];
                            s_crow[at] = __ldcg(a.cand_row + i);
                        }
                    }
                }
            }
            __syncthreads();
            const unsigned int have = min(s_cand, kCutBlockCand);
            for (unsigned int i = tid; i < have; i += kCutThreads) {
                const uint64_t mine = s_ckey[i];
                unsigned int up = 0, same = 0;
                for (unsigned int q = 0; q < have; ++q) {
                    const uint64_t o = s_ckey[q];
                    up += o > mine ? 1u : 0u;
                    same += o == mine ? 1u : 0u;
                }
                if (up < rank && rank <= up + same) {  // (every holder of the boundary agrees)
                    s_bound = mine;
                    s_above = up;
                    s_inbin = same;
                }
            }
            __syncthreads();
            boundary = s_bound + 1;  // as a select key
            const unsigned int quota = rank - s_above, ties = s_inbin;
            nabove = a.keep_n - quota;
            if (quota < ties) {
                // the first `quota` of the boundary's rows stay: which is the last of them?
                for (unsigned int i = tid; i < have; i += kCutThreads) {
                    if (s_ckey[i] != s_bound) continue;
                    unsigned int before = 0;
                    for (unsigned int q = 0; q < have; ++q)
                        before += s_ckey[q] == s_bound && s_crow[q] < s_crow[i] ? 1u : 0u;
                    if (before + 1 == quota) s_tie = s_crow[i];
                }
                __syncthreads();
                last_tie = s_tie;
            }
        }
    }
    if (tid == 0) {
        a.state->boundary = boundary;
        a.state->above = nabove;
        a.state->last_tie = last_tie;
        a.state->status = status;
    }
}

// A warp per tile: positions of its listed partners, each written at its sorted slot.
template <int W, typename T>
__global__ void __launch_bounds__(kPlaceThreads) k_cut_place(const CutArgs<W, T> a, const RotLayer<W> L, uint32_t ntiles,
                                                   uint32_t tpb, CutLive live, uint64_t m,
                                                   uint64_t* __restrict__ Pk, T* __restrict__ Pc,
                                                   uint32_t* __restrict__ pr) {
    __shared__ AmpTab<T> A;
    __shared__ int s_off[kPlaceThreads / 32][kCutRows];
    const int lane = threadIdx.x & 31;
    const unsigned int le = 0xffffffffu >> (31 - lane);
    Ctl* ctl = a.ctl;
    stage_amps<W, T>(L, A);
    __syncthreads();
    const uint32_t SR = a.slot_rows;
    const int NL = a.next.n;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < ntiles; t += warps) {
        const CutTile& ti = a.tiles[t];
        const CutBlock& bl = a.blocks[t / tpb];
        const uint32_t rbase = bl.rbase + ti.rows_before;
        if (lane == 0) {
            pr[t] = rbase;
            if (t == ntiles - 1) pr[ntiles] = rbase + min(__ldg(a.count + t), SR);
        }
        const uint32_t pc = ti.partners;
        if (pc == 0) continue;
        const uint64_t row0 = (uint64_t)t * SR;
        const int base = (int)(bl.pbase + ti.part_before);
        int st[kCutLevels], sp[kCutLevels], en[kCutLevels], sq[kCutLevels];  // carried along, both directions
#pragma unroll
        for (int l = 0; l < kCutLevels; ++l) {
            if (l < NL) {
                const int bp = (int)bl.pbase;
                const int x0 = ti.fwd[l], x1 = ti.fwd[kCutLevels + l];
                const int y0 = ti.bwd[l], y1 = ti.bwd[kCutLevels + l];
                st[l] = x0 >= 0 ? bp + x0 : bl.fwd[l];
                sp[l] = x1 >= 0 ? bp + x1 : bl.fwd[kCutLevels + l];
                const int e = y0 != kCutNone ? bp + y0 : bl.bwd[l];
                en[l] = e == kCutNone ? (int)m : e;
                sq[l] = y1 != kCutNone ? bp + y1 : bl.bwd[kCutLevels + l];
            }
        }
        // backwards over chunks of 32 partners for the first start and split after each, then
        // forwards for the last ones at or before it; the tile's first partner is in the carried
        // prefix (and in its predecessors' suffixes) already
        int* off = s_off[threadIdx.x >> 5];
        // (four chunks' loads in flight)
        constexpr int U = 4;
        const uint32_t chunks = (pc + 31) / 32, steps = (chunks + U - 1) / U;
        for (uint32_t sgl = steps; sgl-- > 0;) {
            uint32_t d[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t j = (sgl * U + u) * 32 + lane;
                d[u] = j > 0 && j < pc ? (uint32_t)a.D[row0 + j] : 0xFFFFu;
            }
#pragma unroll
            for (int u = U - 1; u >= 0; --u) {
                const uint32_t j = (sgl * U + u) * 32 + lane;
                const int at = base + (int)((sgl * U + u) * 32);
                int f = 0;
#pragma unroll
                for (int l = 0; l < kCutLevels; ++l) {
                    if (l < NL) {
                        const uint32_t rk = a.next.rank[l];
                        const unsigned int bs = __ballot_sync(0xffffffffu, d[u] < rk);
                        const unsigned int bp = __ballot_sync(0xffffffffu, d[u] == rk);
                        const unsigned int us = bs & ~le, up = bp & ~le;
                        const int e = us ? at + __ffs(us) - 1 : en[l], q = up ? at + __ffs(up) - 1 : sq[l];
                        if (q < e) f += e - q;
                        if (bs) en[l] = at + __ffs(bs) - 1;
                        if (bp) sq[l] = at + __ffs(bp) - 1;
                    }
                }
                if (j < pc) off[j] = f;
            }
        }
        __syncwarp();
        for (uint32_t sgl = 0; sgl < steps; ++sgl) {
            uint32_t d[U], r[U];
            uint64_t k[U][2 * W];
            T c[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t j = (sgl * U + u) * 32 + lane;
                d[u] = j > 0 && j < pc ? (uint32_t)a.D[row0 + j] : 0xFFFFu;
                r[u] = j < pc ? (uint32_t)a.plist[row0 + j] : 0u;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t j = (sgl * U + u) * 32 + lane;
                c[u] = T(0);
                if (j < pc) {
                    load_key<W>(a.keys, row0 + r[u], k[u]);
                    c[u] = a.coef[row0 + r[u]];
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t j = (sgl * U + u) * 32 + lane;
                const int at = base + (int)((sgl * U + u) * 32);
                const bool on = j < pc;
                int f = on ? off[j] : 0;
#pragma unroll
                for (int l = 0; l < kCutLevels; ++l) {
                    if (l < NL) {
                        const uint32_t rk = a.next.rank[l];
                        const unsigned int bs = __ballot_sync(0xffffffffu, d[u] < rk);
                        const unsigned int bp = __ballot_sync(0xffffffffu, d[u] == rk);
                        const unsigned int ms = bs & le, mp = bp & le;
                        const int s = ms ? at + 31 - __clz(ms) : st[l], p = mp ? at + 31 - __clz(mp) : sp[l];
                        if (p > s) f -= p - s;
                        if (bs) st[l] = at + 31 - __clz(bs);
                        if (bp) sp[l] = at + 31 - __clz(bp);
                    }
                }
                if (!on) continue;
                const long long dest = (long long)base + (long long)j + f;
                if (!PS_GUARD(ctl, dest >= 0 && dest < (long long)m, 1004)) continue;
                const T pcf = live(to_f64(c[u]), (uint32_t)(row0 + r[u])) ? partner_coeff<W, T>(L, A, k[u], c[u]) : T(0);
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    k[u][w] ^= L.gx[w];
                    k[u][W + w] ^= L.gz[w];
                }
                store_key<W>(Pk, (uint64_t)dest, k[u]);
                Pc[dest] = pcf;
            }
        }
    }
}

// Merge-path split points over a cut store: a warp per run of consecutive boundaries.  A split is
// looked for among the slots first (their first rows against the partners), then in its slot.
template <int W>
__global__ void __launch_bounds__(256) k_cut_partition(const uint64_t* __restrict__ Sk, uint64_t n, const CutStore S,
                                                       const uint64_t* __restrict__ Pk, uint64_t m, uint32_t tile_items,
                                                       ulonglong2* __restrict__ bounds, uint4* __restrict__ bslot) {
    const int lane = threadIdx.x & 31;
    const uint32_t num_tiles = (uint32_t)((n + m + tile_items - 1) / tile_items);
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t per = (num_tiles + 1 + warps - 1) / warps;
    const uint32_t first = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per;
    const uint32_t* __restrict__ pr = S.pr;
    uint32_t hint = 0;  // a slot whose first row is not past the split
    for (uint32_t t = first; t <= num_tiles && t < first + per; ++t) {
        uint64_t d = (uint64_t)t * tile_items;
        if (d > n + m) d = n + m;
        const uint64_t lo = d > m ? d - m : 0, hi = d < n ? d : n;  // the split in [lo, hi]
        // the last slot g whose first row is before the split: pr[g] < lo, or pr[g] < hi and that
        // row not after the partner it is paired with on the diagonal
        auto before = [&](uint32_t g) {
            const uint64_t i = pr[g];
            if (i < lo) return true;
            if (i >= hi) return false;
            uint32_t q = g;  // (empty slots share their first row with the next one)
            while (pr[q + 1] == (uint32_t)i) ++q;  // i < hi <= n: some slot holds it
            uint64_t x[2 * W], y[2 * W];
            load_key<W>(Sk, (uint64_t)q * S.slot_rows, x);
            load_key<W>(Pk, d - 1 - i, y);
            return le_regs<W>(x, y);
        };
        uint32_t g0 = hint, g1 = S.tiles;  // answer in [g0, g1)
        if (t > first) {
            // within one tile's items of the last split: a few slots on
            const uint32_t g = g0 + 1 + lane;
            const unsigned int bal = __ballot_sync(0xffffffffu, g < g1 && before(g));
            const int c = __popc(bal);  // a prefix of the lanes
            if (c < 32) {
                g1 = min(g1, g0 + 1 + (uint32_t)c);
                g0 = g0 + (uint32_t)c;
                g1 = g0 + 1;
            } else {
                g0 += 32;
            }
        }
        while (g1 - g0 > 1) {
            const uint32_t span = g1 - g0 - 1;  // candidates g0 + 1 .. g1 - 1
            const uint32_t step = (span + 31) / 32;
            const uint32_t g = g0 + 1 + lane * step;
            const unsigned int bal = __ballot_sync(0xffffffffu, g < g1 && before(g));
            const int c = __popc(bal);
            if (c == 0) {
                g1 = g0 + 1;
            } else {
                const uint32_t nx = g0 + 1 + (uint32_t)c * step;
                g0 = g0 + 1 + (uint32_t)(c - 1) * step;
                g1 = min(g1, nx);
            }
        }
        hint = g0;
        const uint64_t s0 = pr[g0], s1 = pr[g0 + 1];
        uint64_t l = max(lo, s0), h = min(hi, s1);
        if (h < l) h = l;
        auto pred = [&](uint64_t i) {  // row i of slot g0 not after its partner
            uint64_t x[2 * W], y[2 * W];
            load_key<W>(Sk, (uint64_t)g0 * S.slot_rows + (i - s0), x);
            load_key<W>(Pk, d - 1 - i, y);
            return le_regs<W>(x, y);
        };
        while (h - l > 32) {
            const uint64_t span = h - l;
            const unsigned int bal = __ballot_sync(0xffffffffu, pred(l + (span * (uint64_t)lane) / 32));
            const int c = __popc(bal);
            if (c == 0) {
                h = l;
                break;
            }
            const uint64_t p0 = l + (span * (uint64_t)(c - 1)) / 32;
            const uint64_t p1 = c < 32 ? l + (span * (uint64_t)c) / 32 : h;
            l = p0 + 1;
            h = p1;
        }
        const uint64_t span = h - l;
        const unsigned int bal = __ballot_sync(0xffffffffu, (uint64_t)lane < span ? pred(l + lane) : false);
        const uint64_t i = l + (uint64_t)__popc(bal);
        uint64_t j = d - i;
        if (lane == 0) {
            if (i > 0 && j < m) {  // an equal pair stays together
                uint32_t g = g0;
                while (pr[g] > i - 1) --g;
                while (pr[g + 1] <= i - 1) ++g;
                uint64_t x[2 * W], y[2 * W];
                load_key<W>(Sk, (uint64_t)g * S.slot_rows + (i - 1 - pr[g]), x);
                load_key<W>(Pk, j, y);
                if (eq_regs<W>(x, y)) ++j;
            }
            uint32_t g = g0;  // the slot of row i (the last one when i == n)
            while (g + 1 < S.tiles && pr[g + 1] <= i) ++g;
            bounds[t] = make_ulonglong2(i, j);
            bslot[t] = make_uint4(g, pr[g], pr[g + 1], 0u);
        }
        __syncwarp();
    }
}

template <int W, typename T>
int CutOps<W, T>::blocks(int sms) {
    return std::min(2 * (sms > 0 ? sms : 1), kCutThreads);
}

template <int W, typename T>
cudaError_t CutOps<W, T>::configure() {
    return cudaFuncSetAttribute(k_topn_cut<W, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCutSmem);
}

template <int W, typename T>
cudaError_t CutOps<W, T>::cut(const CutArgs<W, T>& a, int sms, cudaStream_t st, KernelProf* prof) {
    prof->begin(K_TOPN_HIST, 0.0, st);
    if (a.slot_rows > kCutRows) return cudaErrorInvalidValue;
    k_topn_cut<W, T><<<blocks(sms), kCutThreads, kCutSmem, st>>>(a);
    prof->end(st);
    return cudaGetLastError();
}

template <int W, typename T>
cudaError_t CutOps<W, T>::place(const CutArgs<W, T>& a, const RotLayer<W>& L, uint32_t tiles, CutLive live, uint64_t m,
                                uint64_t* Pk, T* Pc, uint32_t* pr, int sms, cudaStream_t st, KernelProf* prof) {
    const uint32_t G = (uint32_t)blocks(sms), tpb = (tiles + G - 1) / G;
    const uint32_t grid = std::min<uint32_t>((tiles + kPlaceThreads / 32 - 1) / (kPlaceThreads / 32), 8u * (uint32_t)sms);
    if (a.slot_rows > kCutRows) return cudaErrorInvalidValue;
    prof->begin(K_LEVEL_APPLY, 0.0, st);
    k_cut_place<W, T><<<grid, kPlaceThreads, 0, st>>>(a, L, tiles, tpb, live, m, Pk, Pc, pr);
    prof->end(st);
    return cudaGetLastError();
}

template <int W, typename T>
cudaError_t CutOps<W, T>::partition(const uint64_t* Sk, uint64_t n, const CutStore& S, const uint64_t* Pk, uint64_t m,
                                    uint32_t tile_items, ulonglong2* bounds, uint4* bslot, int sms, cudaStream_t st,
                                    KernelProf* prof) {
    const uint32_t tiles = (uint32_t)((n + m + tile_items - 1) / tile_items);
    const uint32_t grid = std::min<uint32_t>((tiles + 1 + 7) / 8, 8u * (uint32_t)sms);
    prof->begin(K_PARTITION, 0.0, st);
    k_cut_partition<W><<<grid, 256, 0, st>>>(Sk, n, S, Pk, m, tile_items, bounds, bslot);
    prof->end(st);
    return cudaGetLastError();
}

template struct CutOps<1, double>;
template struct CutOps<1, float>;
template struct CutOps<2, double>;
template struct CutOps<2, float>;
template struct CutOps<4, double>;
template struct CutOps<4, float>;

}  // namespace psb
