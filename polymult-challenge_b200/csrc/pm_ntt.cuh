// pm_ntt.cuh -- the register-level pieces of the NTT shared by its passes and by the GEMM kernels
// that run the first (forward) or last (inverse) four column stages: the radix-2^RB butterfly
// networks and the sources of their Shoup twiddles.
//
// Phase k of an NB-bit line covers stage bits NB-1-4k down to b0_k = max(0, NB - 4(k+1));
// its registers hold index bits [b0_k, b0_k + 4) and the thread's position supplies the
// rest (low bits below b0_k, high bits above).  The last phase of a line whose length is
// not a power of 16 re-uses bits [0, 4) and skips the stages an earlier phase has done.
#pragma once

#include "pm_device.cuh"

namespace pm {
namespace {

template <int NB>
struct LineCfg {
    static constexpr int RB = NB < 4 ? NB : 4;      // index bits held in registers
    static constexpr int E = 1 << RB;               // elements per thread
    static constexpr int NPH = RB == 0 ? 0 : (NB + RB - 1) / RB;  // phases (none for a 1-point line)
    __host__ __device__ static constexpr int b0(int k) { return NB - RB * (k + 1) > 0 ? NB - RB * (k + 1) : 0; }
    // first local stage of phase k (local stage t pairs register bit RB-1-t)
    __host__ __device__ static constexpr int t0(int k) { return b0(k) + RB - 1 - (NB - 1 - RB * k); }
    // global stage index of local stage t of phase k: ls = NB - 1 - (b0 + RB - 1 - t)
    __host__ __device__ static constexpr int ls(int k, int t) { return NB - b0(k) - RB + t; }
};

// Forward (CT) radix network on v[] over local stages t0..RB-1 of one phase.  stw(t) returns
// the stage's twiddle source: w[m] is the Shoup-form Tw2 {w, floor(w 2^32 / p)} of group m
// (gi = (hi << t) | m; hi is folded in by stw).
template <int RB, int T0, class StwF>
__device__ __forceinline__ void radix_fwd(uint32_t (&v)[1 << RB], const StwF& stw, uint32_t p) {
#pragma unroll
    for (int t = T0; t < RB; ++t) {
        const int h = (1 << RB) >> (t + 1);
        const auto w = stw(t);
#pragma unroll
        for (int m = 0; m < (1 << t); ++m) {
            const Tw2 wm = w[m];
#pragma unroll
            for (int i = 0; i < h; ++i) {
                bfly_ct_sh(v[m * 2 * h + i], v[m * 2 * h + i + h], wm, p);
            }
        }
    }
}

// The forward network on two operands' lines that share their twiddles (the same prime and
// row): each twiddle is read once for both butterflies.
template <int RB, int T0, class StwF>
__device__ __forceinline__ void radix_fwd2(uint32_t (&v)[1 << RB], uint32_t (&u)[1 << RB], const StwF& stw,
                                           uint32_t p) {
#pragma unroll
    for (int t = T0; t < RB; ++t) {
        const int h = (1 << RB) >> (t + 1);
        const auto w = stw(t);
#pragma unroll
        for (int m = 0; m < (1 << t); ++m) {
            const Tw2 wm = w[m];
#pragma unroll
            for (int i = 0; i < h; ++i) {
                bfly_ct_sh(v[m * 2 * h + i], v[m * 2 * h + i + h], wm, p);
                bfly_ct_sh(u[m * 2 * h + i], u[m * 2 * h + i + h], wm, p);
            }
        }
    }
}

// Inverse (GS) network, local stages RB-1 down to T0, mirrored twiddles from stw(t).
template <int RB, int T0, class StwF>
__device__ __forceinline__ void radix_inv(uint32_t (&v)[1 << RB], const StwF& stw, uint32_t p) {
#pragma unroll
    for (int t = RB - 1; t >= T0; --t) {
        const int h = (1 << RB) >> (t + 1);
        const auto w = stw(t);
#pragma unroll
        for (int m = 0; m < (1 << t); ++m) {
            const Tw2 wm = w[m];
#pragma unroll
            for (int i = 0; i < h; ++i) {
                bfly_gs_sh(v[m * 2 * h + i], v[m * 2 * h + i + h], wm, p);
            }
        }
    }
}

// The inverse network on two lines that share their twiddles.
template <int RB, int T0, class StwF>
__device__ __forceinline__ void radix_inv2(uint32_t (&v)[1 << RB], uint32_t (&u)[1 << RB], const StwF& stw,
                                           uint32_t p) {
#pragma unroll
    for (int t = RB - 1; t >= T0; --t) {
        const int h = (1 << RB) >> (t + 1);
        const auto w = stw(t);
#pragma unroll
        for (int m = 0; m < (1 << t); ++m) {
            const Tw2 wm = w[m];
#pragma unroll
            for (int i = 0; i < h; ++i) {
                bfly_gs_sh(v[m * 2 * h + i], v[m * 2 * h + i + h], wm, p);
                bfly_gs_sh(u[m * 2 * h + i], u[m * 2 * h + i + h], wm, p);
            }
        }
    }
}

// A stage's run of 2^t consecutive Shoup-form twiddles {w, floor(w 2^32 / p)} starting at
// `src`, aligned to 2^t entries.  w[m] is entry m (REV: entry 2^t - 1 - m), read at use as
// half of a 16-byte pair (the two entries of a pair come from one load), so that no more of
// the run than the current butterflies need is held in registers.
template <bool REV>
struct RunTw {
    const uint2* src;
    int n;
    __device__ __forceinline__ Tw2 operator[](int m) const {
        const int e = REV ? n - 1 - m : m;
        if (n == 1) {
            const uint2 u = __ldg(src);
            return Tw2{u.x, u.y};
        }
        const uint4 u = __ldg(reinterpret_cast<const uint4*>(src) + (e >> 1));
        return (e & 1) ? Tw2{u.z, u.w} : Tw2{u.x, u.y};
    }
};

// A column stage's run of 2^t Shoup twiddles in shared memory, starting at `start` (aligned to
// 2^t entries): w[m] is entry m (REV: entry 2^t - 1 - m), read as half of a 16-byte pair.
template <bool REV>
struct SmemRun {
    const Tw2* start;
    int n;
    __device__ __forceinline__ Tw2 operator[](int m) const {
        const int e = REV ? n - 1 - m : m;
        if (n == 1) return start[0];
        const uint4 u = reinterpret_cast<const uint4*>(start)[e >> 1];
        return (e & 1) ? Tw2{u.z, u.w} : Tw2{u.x, u.y};
    }
};

// A stage's 2^t twiddles in a shared-memory table with one row per twiddle and one column per
// prime: w[m] is row m of `src` (REV: row 2^t - 1 - m), `stride` entries apart.  Neighbouring
// primes' entries are neighbours, so that lanes holding different primes read different banks.
template <bool REV>
struct StrideTw {
    const uint2* src;
    int stride, n;
    __device__ __forceinline__ Tw2 operator[](int m) const {
        const uint2 u = src[(REV ? n - 1 - m : m) * stride];
        return Tw2{u.x, u.y};
    }
};

}  // namespace
}  // namespace pm
