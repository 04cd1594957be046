// Device bodies shared by the NTT passes of the three-prime (ntt_kernels.cu)
// and five-prime (wide_kernels.cu) pipelines: butterflies in registers, rounds
// in shared memory, inter-pass twiddles.
#pragma once
#include "engine.h"
#include "pass_common.cuh"

namespace bgpu {

// ---- register-resident butterflies ------------------------------------------

// DIF stages for pair bits HI..LO on the 2^R elements base + (j << LO),
// starting at stage T0 (the stages before it already done by the caller).
// Element pair (i, i+h): (a, b) -> (a+b, (a-b) * omega_{2h}^(i mod h)).
template <bool LAZY, int R, int HI, int LO, int T0 = 0>
__device__ __forceinline__ void dif_regs(uint32_t (&x)[1 << R], uint32_t base_low,
                                         const uint2* __restrict__ tw, uint32_t p) {
    const uint2* twb = tw + base_low;  // every twiddle below is twb[compile-time offset]
#pragma unroll
    for (int t = T0; t < R; ++t) {
        const uint32_t h = 1u << (HI - t);
        const int dist = 1 << (R - 1 - t);
#pragma unroll
        for (int j = 0; j < (1 << R); ++j) {
            if (j & dist) continue;
            if (LO == 0 && (j & (dist - 1)) == 0) {
                Bfly<LAZY>::dif1(x[j], x[j + dist], p);  // omega^0 (base_low is 0 when LO == 0)
            } else {
                const uint2 w = __ldg(twb + h + ((uint32_t)(j & (dist - 1)) << LO));
                Bfly<LAZY>::dif(x[j], x[j + dist], w.x, w.y, p);
            }
        }
    }
}

// DIT stages for pair bits LO..HI (inverse table):
// (a, b) -> (a + b*w, a - b*w), w = omega_{2h}^-(i mod h).
template <bool LAZY, int R, int HI, int LO>
__device__ __forceinline__ void dit_regs(uint32_t (&x)[1 << R], uint32_t base_low,
                                         const uint2* __restrict__ tw, uint32_t p) {
    const uint2* twb = tw + base_low;
#pragma unroll
    for (int t = R - 1; t >= 0; --t) {
        const uint32_t h = 1u << (HI - t);
        const int dist = 1 << (R - 1 - t);
#pragma unroll
        for (int j = 0; j < (1 << R); ++j) {
            if (j & dist) continue;
            if (LO == 0 && (j & (dist - 1)) == 0) {
                Bfly<LAZY>::dit1(x[j], x[j + dist], p);
            } else {
                const uint2 w = __ldg(twb + h + ((uint32_t)(j & (dist - 1)) << LO));
                Bfly<LAZY>::dit(x[j], x[j + dist], w.x, w.y, p);
            }
        }
    }
}

// One smem round (load -> butterflies -> store back); no sync inside.
template <bool LAZY, int L, int C, int T, int K, bool INV>
__device__ __forceinline__ void smem_round(uint32_t* sm, const uint2* __restrict__ tw, uint32_t p,
                                           int tid) {
    using Gr = Group<L, C, K>;
    constexpr int R = Gr::R;
#pragma unroll 2
    for (int g = tid; g < Gr::G; g += T) {
        const Gr gr(g);
        uint32_t x[1 << R];
#pragma unroll
        for (int j = 0; j < (1 << R); ++j) x[j] = sm[gr.at(j)];
        if constexpr (INV)
            dit_regs<LAZY, R, Gr::HI, Gr::LO>(x, gr.base_low, tw, p);
        else
            dif_regs<LAZY, R, Gr::HI, Gr::LO>(x, gr.base_low, tw, p);
#pragma unroll
        for (int j = 0; j < (1 << R); ++j) sm[gr.at(j)] = x[j];
    }
}

// DIF rounds K..KEND in smem, each followed by a block barrier.
template <bool LAZY, int L, int C, int T, int K, int KEND>
__device__ __forceinline__ void dif_rounds(uint32_t* sm, const uint2* tw, uint32_t p, int tid) {
    if constexpr (K <= KEND) {
        smem_round<LAZY, L, C, T, K, false>(sm, tw, p, tid);
        __syncthreads();
        dif_rounds<LAZY, L, C, T, K + 1, KEND>(sm, tw, p, tid);
    }
}

// DIT rounds K down to KEND in smem, each followed by a barrier.
template <bool LAZY, int L, int C, int T, int K, int KEND>
__device__ __forceinline__ void dit_rounds(uint32_t* sm, const uint2* tw, uint32_t p, int tid) {
    if constexpr (K >= KEND) {
        smem_round<LAZY, L, C, T, K, true>(sm, tw, p, tid);
        __syncthreads();
        dit_rounds<LAZY, L, C, T, K - 1, KEND>(sm, tw, p, tid);
    }
}

// omega_N^(+-e) as a fully reduced Montgomery form from the two split tables.
__device__ __forceinline__ uint32_t inter_twiddle(const NttConsts& c, int q, int dir, uint32_t e,
                                                  int log_n, uint32_t p) {
    const uint32_t em = e << (c.log_max - log_n);
    const uint32_t hi = __ldg(&c.th[q][dir][em >> c.split].x);
    const uint2 lo = __ldg(&c.tl[q][dir][em & ((1u << c.split) - 1u)]);
    return mont_mul_pre(hi, lo.x, lo.y, p);
}

// x * omega (omega from inter_twiddle), lazily (0, 2p) or strictly [0, p).
template <bool LAZY>
__device__ __forceinline__ uint32_t twiddle_mul(uint32_t x, uint32_t w, uint32_t p, uint32_t pinv) {
    const uint32_t r = mont_lazy(x, w, w * pinv, p);
    return LAZY ? r : csub(r, p);
}

// x * S * B for Montgomery pairs S = (w, w') and B = (bw, bw'): the
// inter-pass twiddle split as a per-CTA power table entry times a per-group
// factor, lazily (0, 2p) or strictly [0, p).
template <bool LAZY>
__device__ __forceinline__ uint32_t mul2(uint32_t x, uint2 sp, uint32_t bw, uint32_t bwp,
                                         uint32_t p) {
    const uint32_t y = mont_lazy(mont_lazy(x, sp.x, sp.y, p), bw, bwp, p);
    return LAZY ? y : csub(y, p);
}

__host__ __device__ constexpr uint32_t brev_c(uint32_t v, int bits) {
    uint32_t r = 0;
    for (int i = 0; i < bits; ++i) r |= ((v >> i) & 1u) << (bits - 1 - i);
    return r;
}

__device__ __forceinline__ uint32_t bitrev(uint32_t v, int bits) {
    return bits == 0 ? 0u : (__brev(v) >> (32 - bits));
}

// a*b*2^-32 mod p in [0, p); the 2^-32 and the inverse transform's N^-1 are
// both cancelled by the scale N^-1 * 2^32 folded into the row's inverse
// inter-pass twiddle (one multiply per group instead of one per point).
template <bool LAZY>
__device__ __forceinline__ uint32_t pointwise(uint32_t a, uint32_t b, uint32_t p, uint32_t pinv) {
    if constexpr (LAZY)
        return csub(mont_lazy(a, b, b * pinv, p), p);  // a, b < 2p, 4p < 2^32: product term < p
    else
        return mont_mul(a, b, p, pinv);
}

// Thread number within a row's group of T threads: the CTA's own thread
// number when the CTA is one group (MULTI false: the compiler re-reads it
// instead of holding a computed copy in a register), else the position in
// its group (a CTA holding several rows of a mixed-length launch).
template <int T, bool MULTI>
__device__ __forceinline__ int sub_tid() {
    return MULTI ? (int)(threadIdx.x & (T - 1)) : (int)threadIdx.x;
}

// DIF of one row: round 0 from global into smem, then rounds 1..nr-2 (the
// last round is done by mid_turn).
template <bool LAZY, int L1, int T, bool MULTI>
__device__ __forceinline__ void mid_dif_row(const uint32_t* row, uint32_t* s, const uint2* twf,
                                            uint32_t p) {
    const int tid = sub_tid<T, MULTI>();
    using P1 = Plan<L1>;
    using Gr = Group<L1, 1, 0>;
    constexpr int R = Gr::R;
#pragma unroll 2
    for (int g = tid; g < Gr::G; g += T) {
        const Gr gr(g);
        uint32_t x[1 << R];
#pragma unroll
        for (int j = 0; j < (1 << R); ++j) x[j] = row[gr.idx(j)];
        dif_regs<LAZY, R, Gr::HI, Gr::LO>(x, gr.base_low, twf, p);
#pragma unroll
        for (int j = 0; j < (1 << R); ++j) s[gr.at(j)] = x[j];
    }
    __syncthreads();
    dif_rounds<LAZY, L1, 1, T, 1, P1::nr - 2>(s, twf, p, tid);
}

}  // namespace bgpu
