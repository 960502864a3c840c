// ps_rotlayer.cuh -- device helpers of a rotation layer's table shared by the layer kernels,
// the kernel that runs many layers in one launch and the TopN compaction that classifies its
// output rows for the next layer: support pattern of a key, per-pattern amplitudes staged in
// shared memory, the partner test, own and partner coefficients, folded noise, divergence rank,
// merge comparisons.  LT: RotLayer<W>, or a type with its fields.
#pragma once

#include <type_traits>

#include "ps_device.cuh"
#include "ps_kernels.h"

namespace psb {

// word `wi` of a key held in registers, by an unrolled select (a runtime index into a
// register array would move the array to local memory)
template <int W>
__device__ __forceinline__ uint64_t pick(const uint64_t* k, int wi) {
    uint64_t v = k[0];
#pragma unroll
    for (int w = 1; w < 2 * W; ++w) v = (w == wi) ? k[w] : v;
    return v;
}

// support pattern of key k (LocalPtm::support_bits, channel/prepared.rs:141-151)
template <int W, typename LT>
__device__ __forceinline__ uint32_t pattern_of(const LT& L, const uint64_t* k) {
    uint32_t s = (uint32_t)((pick<W>(k, L.qw[0]) >> L.qb[0]) & 1u) |
                 (uint32_t)((pick<W>(k, W + L.qw[0]) >> L.qb[0]) & 1u) << 1 |
                 (uint32_t)((pick<W>(k, L.qw[1]) >> L.qb[1]) & 1u) << 2 |
                 (uint32_t)((pick<W>(k, W + L.qw[1]) >> L.qb[1]) & 1u) << 3;
    return s & L.pattern_mask;
}

template <typename T>
struct Amp;
template <>
struct Amp<double> {
    template <int W>
    __device__ static double a0(const RotLayer<W>& L, uint32_t s) { return L.a0[s]; }
    template <int W>
    __device__ static double a1(const RotLayer<W>& L, uint32_t s) { return L.a1[s]; }
    template <typename LT>
    __device__ static double cs(const LT& L) { return L.cos64; }
    template <typename LT>
    __device__ static double sn(const LT& L) { return L.sin64; }
};
template <>
struct Amp<float> {
    template <int W>
    __device__ static float a0(const RotLayer<W>& L, uint32_t s) { return L.a0f[s]; }
    template <int W>
    __device__ static float a1(const RotLayer<W>& L, uint32_t s) { return L.a1f[s]; }
    template <typename LT>
    __device__ static float cs(const LT& L) { return L.cos32; }
    template <typename LT>
    __device__ static float sn(const LT& L) { return L.sin32; }
};

// The layer's per-pattern amplitudes staged in shared memory: indexing the kernel-parameter
// copy with a per-lane pattern would serialize on the constant cache.
template <typename T>
struct AmpTab {
    T a0[16];
    T a1[16];
};

template <int W, typename T>
__device__ __forceinline__ void stage_amps(const RotLayer<W>& L, AmpTab<T>& t) {
    if (threadIdx.x < 16) {
        t.a0[threadIdx.x] = Amp<T>::a0(L, threadIdx.x);
        t.a1[threadIdx.x] = Amp<T>::a1(L, threadIdx.x);
    }
}

template <int W, typename T, typename LT>
__device__ __forceinline__ bool emits_partner_regs(const LT& L, const AmpTab<T>& A,
                                                   const uint64_t (&k)[2 * W]) {
    if (L.wide == 1) {
        uint64_t f = 0;
#pragma unroll
        for (int i = 0; i < W; ++i) f ^= (k[i] & L.gz[i]) ^ (k[W + i] & L.gx[i]);
        return (__popcll(f) & 1) != 0;
    }
    return A.a1[pattern_of<W>(L, k)] != T(0);
}

template <int W>
__device__ __forceinline__ uint32_t div_regs(const uint64_t (&a)[2 * W], const uint64_t (&b)[2 * W]) {
    uint32_t r = 0xFFFFu;
#pragma unroll
    for (int i = 2 * W - 1; i >= 0; --i) {
        uint64_t d = a[i] ^ b[i];
        if (d) r = 64u * i + (uint32_t)__clzll((long long)d);
    }
    return r;
}

// Own-row coefficient after the layer.
template <int W, typename T, typename LT>
__device__ __forceinline__ T own_coeff(const LT& L, const AmpTab<T>& A, const uint64_t* k, T c) {
    if (L.wide) {
        if (L.wide == 1) return anticommutes<W>(k, L.gx, L.gz) ? mul_rn(c, Amp<T>::cs(L)) : c;
        const T a = A.a0[pattern_of<W>(L, k)];  // a moved row leaves nothing, whatever its coefficient
        return a == T(0) ? T(0) : mul_rn(c, a);
    }
    return mul_rn(c, A.a0[pattern_of<W>(L, k)]);
}

// Partner coefficient (DeltaEntry::emit / PreparedRotation::emit_generator).
template <int W, typename T, typename LT>
__device__ __forceinline__ T partner_coeff(const LT& L, const AmpTab<T>& A, const uint64_t* k, T c) {
    if (L.wide == 1) {
        uint32_t total = (1u + product_phase<W>(k, L.gx, L.gz)) & 3u;
        T m = (total & 2u) ? -c : c;  // real mul_phase, coefficient.rs:107-114
        return mul_rn(m, Amp<T>::sn(L));
    }
    return mul_rn(c, A.a1[pattern_of<W>(L, k)]);
}

// The folded noise channels, staged in shared memory (their factors are indexed by each lane's
// pattern).
template <typename T>
struct NoiseSmem {
    T f[kMaxNoise][4];
    uint16_t q[kMaxNoise];
    int n;
};

template <typename T>
__device__ __forceinline__ void stage_noise(const NoiseList& N, NoiseSmem<T>& S) {
    for (int i = threadIdx.x; i < N.n * 4; i += blockDim.x) {
        if constexpr (std::is_same<T, double>::value)
            S.f[i >> 2][i & 3] = N.f[i >> 2][i & 3];
        else
            S.f[i >> 2][i & 3] = N.ff[i >> 2][i & 3];
    }
    for (int i = threadIdx.x; i < N.n; i += blockDim.x) S.q[i] = N.q[i];
    if (threadIdx.x == 0) S.n = N.n;
}

// The folded channels applied to coefficient v of key k in order, as the separate layers would:
// a channel multiplies by its factor for k's pattern on its qubit (the identity's factor is 1,
// skipped), then the term must stay nonzero and pass the keep program.  Returns the index of the
// channel after which the term is dropped, or S.n when it survives all of them.
template <int W, typename T>
__device__ __forceinline__ int noise_apply(const NoiseSmem<T>& S, const KeepProg& keep, const uint64_t* k, T& v) {
    if (!(v != T(0) && keep_eval<W>(keep, k, to_f64(v)))) return 0;
    for (int j = 0; j < S.n; ++j) {
        const int q = S.q[j];
        const uint32_t s = (uint32_t)((pick<W>(k, q >> 6) >> (q & 63)) & 1u) |
                           (uint32_t)((pick<W>(k, W + (q >> 6)) >> (q & 63)) & 1u) << 1;
        if (s) {
            v = mul_rn(v, S.f[j][s]);
            if (!(v != T(0) && keep_eval<W>(keep, k, to_f64(v)))) return j;
        }
    }
    return S.n;
}

// Rows of a staged run in shared memory and comparisons on keys held in registers.
template <int W>
__device__ __forceinline__ void ld_row(const uint64_t* base, uint32_t r, uint64_t (&k)[2 * W]) {
    const ulonglong2* p = reinterpret_cast<const ulonglong2*>(base + (size_t)r * 2 * W);
#pragma unroll
    for (int q = 0; q < W; ++q) {
        ulonglong2 v = p[q];
        k[2 * q] = v.x;
        k[2 * q + 1] = v.y;
    }
}

template <int W>
__device__ __forceinline__ bool le_regs(const uint64_t (&a)[2 * W], const uint64_t (&b)[2 * W]) {
#pragma unroll
    for (int i = 0; i < 2 * W; ++i)
        if (a[i] != b[i]) return a[i] < b[i];
    return true;
}
template <int W>
__device__ __forceinline__ bool eq_regs(const uint64_t (&a)[2 * W], const uint64_t (&b)[2 * W]) {
    uint64_t d = 0;
#pragma unroll
    for (int i = 0; i < 2 * W; ++i) d |= a[i] ^ b[i];
    return d == 0;
}

}  // namespace psb
