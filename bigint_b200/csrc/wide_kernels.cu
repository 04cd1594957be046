// Wide-digit NTT product pipeline (see wide.h): five, six or seven primes,
//   1. k_wide_fwd   per (8-column tile, prime, operand): digits reduced mod p, length-N2 DIF over
//                   n2, times omega_N^(n1 k2)
//   2. k_wide_rows  per (row, prime): length-N1 DIF of A's and B's row, pointwise product, DIT back,
//                   times omega_N^-(n1 k2) and the scale, in place
//   3. k_wide_inv   per (8-column tile, prime): length-N2 DIT, in place, to natural order
//   4. k_wide_carry CRT of the residues, sums of chunks of four digits and the carry scan
// or, up to 2^12 points, k_wide_short in place of 1 to 3.
// The transforms are those of ntt_kernels.cu.  The CRT is not Garner's: the
// scale of the row pass carries (M/p)^-1, so a coefficient is a sum of
// residue-by-constant products less a multiple q of M found in single
// precision (five primes: 20 wide multiply-adds); it runs in the carry kernel,
// so no chunk sums go through memory.
// 2^24 x 2^24 bits (2^19 points): 63.7 us on three primes, 46.2 here; the
// multiply pipe is 47 to 52 % busy in the forward and row passes of one cold
// product, 27 % in the inverse pass, issue slots 34 to 48 %.
#include <cstring>

#include "carry_common.cuh"
#include "ntt_bodies.cuh"
#include "wide.h"

namespace bgpu {

constexpr int kWideCols = 8;
// Threads of the column passes: the groups of a round (8 columns of 2^L2 / 8 or
// 2^L2 / 16), so that short columns leave no thread idle: forward and inverse
// pass per 2^19 points of a batch, columns of 2^6 rows 28.0 + 10.8 -> 14.2 + 5.5 us,
// of 2^8 rows 16.8 + 9.1 -> 13.3 + 5.2 us against 256 threads throughout.
// Columns of 2^11 rows (64 KB tiles, two or three a SM) run two CTAs of 512
// threads forward and three of 256 inverse: 2^24 points 548 + 249 us against
// 647 + 249 (256 x 3) and 548 + 265 (512 x 2), and 587 + 452 with the
// compiler's registers at 256 threads.
__host__ __device__ constexpr int wide_col_threads(int l2, bool fwd) {
    return l2 <= 5 ? 32 : l2 <= 7 ? 64 : l2 == 8 ? 128 : l2 == 11 && fwd ? 512 : 256;
}
// Row pass: threads of a row and rows of a CTA.  Short rows have fewer groups
// than a warp has lanes (16 at 2^8 points), so a CTA takes several side by
// side: per 2^19 points of a batch, rows of 2^8 points 23.5 -> 12.7 us, of 2^7
// points 34.8 -> 11.7 us, of 2^6 42.6 -> 11.3 us against one 32-thread CTA a row.
__host__ __device__ constexpr int wide_row_threads(int l1) {
    return l1 >= 12 ? 256 : l1 >= 9 ? (1 << (l1 - 4)) : l1 == 8 ? 16 : 8;
}
__host__ __device__ constexpr int wide_rows_per_cta(int l1) { return l1 >= 10 ? 1 : 128 / wide_row_threads(l1); }
// Rows of 2^13 points and more of a product of two operands use one row buffer:
// A's transform is parked in its own plane and read back by the pointwise
// product, so that four and three CTAs share an SM instead of three and one.
// Row pass, two buffers -> one: 2^23 points in rows of 2^13 358 -> 334 us, 2^25
// points in rows of 2^14 1807 (512 threads) -> 1407 us; rows of 2^12 points are
// faster with two (2^21 points 81 against 88 us).
__host__ __device__ constexpr bool wide_one_buffer(int l1) { return l1 >= 13; }
// Shared words of a row: its buffers and 16 Shoup pairs, a warp's rows in different banks.
__host__ __device__ constexpr uint32_t wide_row_words(int l1, bool square) {
    return ((square || wide_one_buffer(l1) ? 1u : 2u) << l1) + 32u + (l1 >= 10 ? 0u : (uint32_t)wide_row_threads(l1) % 32u);
}

// lazy and strict sets of five, six and seven primes
constexpr int kWideSets = kNumSets - kFirstWideSet;
__constant__ NttConsts c_wide[kWideSets];
__constant__ WideCrt c_crt[kWideSets];
__constant__ uint32_t c_scale[kWideSets][kWideMaxLogN + 1][kWideMaxPrimes];  // row pass, Montgomery form
__host__ __device__ constexpr int wide_set_index(int np, bool lazy) { return 2 * (np - kWidePrimes) + (lazy ? 0 : 1); }

// Planes of product i.
__device__ __forceinline__ uint32_t* wide_planes(const WideArgs& a, uint32_t i) {
    return a.descs ? a.descs[i].y : a.y + (((size_t)i * (uint32_t)(a.nops * a.np)) << a.log_n);
}

// (hi 2^32 + lo + k p) / 2^32 with the k that clears the low word: one wide
// multiply-add with a 64-bit addend.
__device__ __forceinline__ uint32_t redc(uint32_t lo, uint32_t hi, uint32_t p, uint32_t np) {
    uint32_t r;
    asm("{.reg .u32 z;\n\t"
        "mad.lo.cc.u32 z, %1, %2, %3;\n\t"
        "madc.hi.u32 %0, %1, %2, %4;}"
        : "=r"(r)
        : "r"(lo * np), "r"(p), "r"(lo), "r"(hi));
    return r;
}
// a w 2^-32 mod p, below 2p for any 32-bit a and w < p (np = -p^-1 mod 2^32).
__device__ __forceinline__ uint32_t mont(uint32_t a, uint32_t w, uint32_t p, uint32_t np) {
    const uint64_t t = (uint64_t)a * w;
    return redc((uint32_t)t, (uint32_t)(t >> 32), p, np);
}
// Shoup pair (w, floor(w 2^32 / p)) of w, given r = w 2^32 mod p: the quotient
// is (w 2^32 - r) / p = -r / p mod 2^32.
__device__ __forceinline__ uint2 shoup_of(uint32_t r, uint32_t p, uint32_t np) {
    return make_uint2(csub(redc(r, 0, p, np), p), r * np);
}
// x s b for Shoup pairs: lazily below 2p, or below p for the strict set.
template <bool LAZY>
__device__ __forceinline__ uint32_t shoup2(uint32_t x, uint2 s, uint2 b, uint32_t p) {
    const uint32_t y = shoup_lazy(shoup_lazy(x, s.x, s.y, p), b.x, b.y, p);
    return LAZY ? y : csub(y, p);
}

// ---- 1: forward columns -----------------------------------------------------------

// 32-bit word w of an operand of 28-bit digits (0 beyond its length).
__device__ __forceinline__ uint32_t load_word28(const OperandDesc& in, uint64_t w) {
    const uint32_t* d = static_cast<const uint32_t*>(in.ptr);
    const uint64_t bit = w * 32;
    const uint32_t i = (uint32_t)(bit / 28), sh = (uint32_t)(bit - (uint64_t)i * 28);  // sh in {0, 4, ..., 24}
    uint32_t v = i < in.nsrc ? __ldg(d + i) >> sh : 0u;
    if (i + 1 < in.nsrc) v |= __ldg(d + i + 1) << (28 - sh);
    return v;
}

// Digit n of an operand (0 beyond its nd digits): its words, the unused ones 0.
template <int NP, bool LIMB>
__device__ __forceinline__ void load_digit(const OperandDesc& in, uint32_t nd, uint32_t n, uint32_t (&d)[3]) {
    d[0] = d[1] = d[2] = 0;
    if (n >= nd) return;
    if constexpr (NP == 5 && LIMB) {
        const uint64_t v = __ldg(static_cast<const unsigned long long*>(in.ptr) + n);
        d[0] = (uint32_t)v, d[1] = (uint32_t)(v >> 32);
    } else {
        const uint64_t w = ((uint64_t)n * wide_bits(NP)) >> 5;
        constexpr int NW = NP == 5 ? 2 : 3;
        if constexpr (LIMB) {
            const uint32_t* x = static_cast<const uint32_t*>(in.ptr);
            const uint64_t words = 2 * (uint64_t)in.nsrc;
#pragma unroll
            for (int k = 0; k < NW; ++k)
                if (k == 0 || w + k < words) d[k] = __ldg(x + w + k);
        } else {
#pragma unroll
            for (int k = 0; k < NW; ++k) d[k] = load_word28(in, w + k);
        }
        if constexpr (NP == 6) {  // 80 bits from an even or an odd half word
            const uint32_t sh = (n & 1u) * 16u;
            d[0] = __funnelshift_r(d[0], d[1], sh);
            d[1] = __funnelshift_r(d[1], d[2], sh);
            d[2] = (d[2] >> sh) & 0xffffu;
        }
    }
}

// Round 0: rows n2 = base + (j << LO) read from the operand.  A digit of
// two words becomes digit 2^-32 mod p, of three digit 2^-64 mod p (the scale of
// the row pass undoes it), in [0, 2p) or [0, p).  HALF: the rows of the upper half of the transform are zero; they
// are not loaded and the first stage is one multiply per pair.
template <bool LAZY, int L2, int C, int T, int NP, bool LIMB, bool HALF>
__device__ __forceinline__ void wide_round0(int log_n1, const OperandDesc& in, uint32_t nd, const NttConsts& c, int q,
                                            uint32_t c0, uint32_t* sm, int tid) {
    using Gr = Group<L2, C, 0>;
    constexpr int R = Gr::R;
    constexpr int D = 1 << (R - 1);
    constexpr int NL = HALF ? D : (1 << R);
    const uint32_t p = c.pr[q].p, np = 0u - c.pr[q].pinv, red = c.red[q];
    const uint2* tw = c.stage[q][0];
    const uint32_t stride = 1u << (Gr::LO + log_n1);
#pragma unroll 2
    for (int g = tid; g < Gr::G; g += T) {
        const Gr gr(g);
        uint32_t x[1 << R];
        uint32_t any = 0;
        uint32_t n = c0 + gr.col + (gr.base << log_n1);
#pragma unroll
        for (int j = 0; j < NL; ++j, n += stride) {
            uint32_t d[3];
            load_digit<NP, LIMB>(in, nd, n, d);
            any |= d[0] | d[1] | d[2];
            d[1] -= __umulhi(d[1], red) * p;  // [0, 2p)
            if (!LAZY) d[1] = csub(d[1], p);
            uint32_t r = redc(d[0], d[1], p, np);  // one p more
            if constexpr (NP > 5) {
                if (NP == 7) {  // 80-bit digits have 16 bits here
                    d[2] -= __umulhi(d[2], red) * p;
                    if (!LAZY) d[2] = csub(d[2], p);
                }
                r = redc(r, d[2], p, np);  // below d[2] + p + 1
            }
            x[j] = LAZY ? csub(r, 2 * p) : csub(r, p);
        }
        if (any) {
            if constexpr (HALF) {
                const uint2* twb = tw + gr.base_low;
#pragma unroll
                for (int j = 0; j < D; ++j) {
                    const uint2 w = __ldg(twb + (1u << Gr::HI) + ((uint32_t)j << Gr::LO));
                    const uint32_t t = shoup_lazy(x[j], w.x, w.y, p);
                    x[j + D] = LAZY ? t : csub(t, p);
                }
                dif_regs<LAZY, R, Gr::HI, Gr::LO, 1>(x, gr.base_low, tw, p);
            } else {
                dif_regs<LAZY, R, Gr::HI, Gr::LO>(x, gr.base_low, tw, p);
            }
        } else {
#pragma unroll
            for (int j = 0; j < (1 << R); ++j) x[j] = 0;
        }
#pragma unroll
        for (int j = 0; j < (1 << R); ++j) sm[gr.at(j)] = x[j];
    }
}

template <bool LAZY, int L2, int C, int T, int NP>
__device__ __forceinline__ void wide_load(int log_n1, const OperandDesc& in, size_t nn, const NttConsts& c, int q,
                                          uint32_t c0, uint32_t* sm, int tid) {
    const uint32_t nd = wide_digits(NP, in.nd32);
    const bool half = 2 * (size_t)nd <= nn;
    if (in.fmt == kFmtLimb64) {
        if (half)
            wide_round0<LAZY, L2, C, T, NP, true, true>(log_n1, in, nd, c, q, c0, sm, tid);
        else
            wide_round0<LAZY, L2, C, T, NP, true, false>(log_n1, in, nd, c, q, c0, sm, tid);
    } else {
        if (half)
            wide_round0<LAZY, L2, C, T, NP, false, true>(log_n1, in, nd, c, q, c0, sm, tid);
        else
            wide_round0<LAZY, L2, C, T, NP, false, false>(log_n1, in, nd, c, q, c0, sm, tid);
    }
}

__device__ __forceinline__ OperandDesc wide_operand(const WideFwdArgs& fa, uint32_t product, int op) {
    if (fa.w.descs) return fa.w.descs[product].op[op];
    OperandDesc in = op == 0 ? fa.op[0] : fa.op[1];
    in.ptr = static_cast<const char*>(in.ptr) + (int64_t)product * (op == 0 ? fa.step_a : fa.step_b);
    return in;
}

// CTAs per SM (register caps): 1024 threads' worth of 64 registers, except
// columns of 2^9 rows at 1280 (2^19 points of a batch: 15.0 + 5.7 us; at 1024
// 15.5 + 6.2, at 2048 15.1 + 5.9), of 2^8 rows nine CTAs, and the inverse pass's
// tiles of 2^11 rows.  Nine CTAs (here, and for rows of 2^11 points) hold the 1280
// CTAs of a 2^19-point inverse pass over five primes in one wave; us per product,
// eight -> nine: 2^14 to 2^16 points 11.9 -> 12.0, 15.1 -> 15.1, 16.6 -> 16.6, 2^18
// 29.1 -> 28.7, 2^19 47.7 -> 46.4 (ten 47.2), 2^20 89.4 -> 89.2, 2^21 174.8 ->
// 175.1; 2^18 over six primes 36.8 -> 37.4, over seven 39.1 -> 39.4, 2^19 61.7 -> 61.8;
// per 2^19 points of a batch, 2^14 to 2^20 points, 0.1 to 0.2 less.
__host__ __device__ constexpr int wide_col_blocks(int l2, bool fwd) {
    return l2 == 8 ? 9 : l2 == 9 ? 5 : l2 == 11 && !fwd ? 3 : 1024 / wide_col_threads(l2, fwd);
}

template <bool LAZY, int L2, int T, int NP>
__global__ void __launch_bounds__(T, wide_col_blocks(L2, true)) k_wide_fwd(const WideFwdArgs fa) {
    const WideArgs& a = fa.w;
    using P2 = Plan<L2>;
    constexpr int NR = P2::nr, RL = P2::r(NR - 1), SROW = (1 << RL) + 1;
    static_assert(NR > 1, "column passes of several rounds");
    extern __shared__ __align__(16) uint32_t sm[];  // [2^L2][8] and the column powers
    const NttConsts& c = c_wide[wide_set_index(NP, LAZY)];
    const int q = blockIdx.y, op = (int)(blockIdx.z % (uint32_t)a.nops);
    const uint32_t product = blockIdx.z / (uint32_t)a.nops;
    const uint32_t p = c.pr[q].p, np = 0u - c.pr[q].pinv;
    const uint2* tw = c.stage[q][0];
    const OperandDesc in = wide_operand(fa, product, op);
    const uint32_t c0 = blockIdx.x * kWideCols;
    const size_t nn = (size_t)1 << a.log_n;
    uint32_t* y = wide_planes(a, product) + ((size_t)op * NP + q) * nn;

    // The last round's groups hold slots base + j of one column n1, whose
    // inter-pass twiddle is omega_N^(n1 bitrev(base)) S^bitrev(j): sS[col][m]
    // holds S^m = omega_N^(n1 m 2^(L2-RL)), rows padded against bank conflicts.
    uint2* sS = reinterpret_cast<uint2*>(sm + (kWideCols << L2));
    for (int t = threadIdx.x; t < (kWideCols << RL); t += T) {
        const uint32_t col = (uint32_t)t >> RL, m = (uint32_t)t & ((1u << RL) - 1u);
        sS[col * SROW + m] = shoup_of(
            inter_twiddle(c, q, 0, (((c0 + col) * m) << (L2 - RL)) & (uint32_t)(nn - 1), a.log_n, p), p, np);
    }
    pdl_wait();
    wide_load<LAZY, L2, kWideCols, T, NP>(a.log_n1, in, nn, c, q, c0, sm, threadIdx.x);
    __syncthreads();
    dif_rounds<LAZY, L2, kWideCols, T, 1, NR - 2>(sm, tw, p, threadIdx.x);
    using Gr = Group<L2, kWideCols, NR - 1>;
#pragma unroll 2
    for (int g = threadIdx.x; g < Gr::G; g += T) {
        const Gr gr(g);
        uint32_t x[1 << RL];
#pragma unroll
        for (int j = 0; j < (1 << RL); ++j) x[j] = sm[gr.at(j)];
        dif_regs<LAZY, RL, Gr::HI, Gr::LO>(x, gr.base_low, tw, p);
        const uint32_t n1 = c0 + gr.col;
        const uint2 bw = shoup_of(
            inter_twiddle(c, q, 0, (n1 * bitrev(gr.base, L2)) & (uint32_t)(nn - 1), a.log_n, p), p, np);
        const uint2* srow = sS + gr.col * SROW;
#pragma unroll
        for (int j = 0; j < (1 << RL); ++j)
            y[((size_t)gr.idx(j) << a.log_n1) + n1] = shoup2<LAZY>(x[j], srow[brev_c(j, RL)], bw, p);
    }
    pdl_trigger();  // late: an early trigger parks row-pass CTAs on SMs this pass still fills
}

// ---- 2: rows -----------------------------------------------------------------------

// CTAs per SM: 1024 threads' worth of 64 registers; rows of 2^8 points, which
// spill there, five CTAs of 128 threads (14.1 -> 12.7 us per 2^19 points), of 2^9
// points six, of 2^11 points nine (as the columns above), of 2^14 points three of 80 registers (1407 us at 2^25 points; two
// of 512 threads 1488).
__host__ __device__ constexpr int wide_row_blocks(int l1) {
    return l1 == 8 ? 5 : l1 == 9 ? 6 : l1 == 11 ? 9 : l1 == 13 ? 4 : l1 == 14 ? 3 : 1024 / (wide_row_threads(l1) * wide_rows_per_cta(l1));
}

template <bool LAZY, int L1, bool SQR>
__global__ void __launch_bounds__(wide_row_threads(L1) * wide_rows_per_cta(L1), wide_row_blocks(L1))
    k_wide_rows(const WideArgs a) {
    constexpr int T = wide_row_threads(L1);
    constexpr bool MULTI = wide_rows_per_cta(L1) > 1;
    constexpr bool ONE = !SQR && wide_one_buffer(L1);
    using P1 = Plan<L1>;
    constexpr int NR = P1::nr;
    constexpr int R0 = P1::r(0), LO0 = P1::lo(0);
    static_assert(NR > 1, "rows of several rounds");
    extern __shared__ __align__(16) uint32_t sm[];  // per row: A's row, B's, the powers
    const NttConsts& c = c_wide[a.set];
    const uint32_t sub = MULTI ? threadIdx.x / T : 0u;
    uint32_t* sa = sm + sub * wide_row_words(L1, SQR);
    uint32_t* sb = ONE ? sa : sa + (1u << L1);
    uint2* sT = reinterpret_cast<uint2*>(sa + ((SQR || ONE ? 1u : 2u) << L1));
    const int q = blockIdx.y, tid = sub_tid<T, MULTI>();
    const uint32_t slot = blockIdx.x * wide_rows_per_cta(L1) + sub;
    const uint32_t p = c.pr[q].p, np = 0u - c.pr[q].pinv;
    const uint2* twf = c.stage[q][0];
    const uint2* twi = c.stage[q][1];
    const size_t nn = (size_t)1 << a.log_n;
    uint32_t* row_a = wide_planes(a, blockIdx.z) + q * nn + ((size_t)slot << L1);
    const uint32_t* row_b = row_a + a.np * nn;
    const uint32_t k2 = bitrev(slot, a.log_n - L1);
    const uint32_t scale = c_scale[a.set][a.log_n][q];

    // The last DIT round's groups hold n1 = base + (j << LO0): twiddle
    // omega_N^-(k2 base) sT[j], sT[j] = omega_N^-(k2 j << LO0).
    for (int t = tid; t < (1 << R0); t += T)
        sT[t] = shoup_of(inter_twiddle(c, q, 1, ((k2 * (uint32_t)t) << LO0) & (uint32_t)(nn - 1), a.log_n, p), p, np);
    __syncthreads();
    pdl_wait();

    mid_dif_row<LAZY, L1, T, MULTI>(row_a, sa, twf, p);
    if constexpr (ONE) {  // A's last DIF round, each group's outputs parked in its plane
        using Gr = Group<L1, 1, NR - 1>;
        static_assert(Gr::LO == 0 && Gr::R >= 2, "a group is a run of elements");
#pragma unroll 1
        for (int g = tid; g < Gr::G; g += T) {
            const Gr gr(g);
            uint32_t x[1 << Gr::R];
#pragma unroll
            for (int j = 0; j < (1 << Gr::R); ++j) x[j] = sa[gr.at(j)];
            dif_regs<LAZY, Gr::R, Gr::HI, Gr::LO>(x, gr.base_low, twf, p);
            uint4* o = reinterpret_cast<uint4*>(row_a + gr.base);
#pragma unroll
            for (int j = 0; j < (1 << Gr::R); j += 4) o[j / 4] = make_uint4(x[j], x[j + 1], x[j + 2], x[j + 3]);
        }
        __syncthreads();  // the buffer takes B
        mid_dif_row<LAZY, L1, T, MULTI>(row_b, sb, twf, p);
    } else if constexpr (!SQR) {
        smem_round<LAZY, L1, 1, T, NR - 1, false>(sa, twf, p, tid);  // A's last DIF round
        mid_dif_row<LAZY, L1, T, MULTI>(row_b, sb, twf, p);
    }
    {  // the last DIF round of B (or A), the pointwise product, the first DIT round
        using Gr = Group<L1, 1, NR - 1>;
        constexpr int R = Gr::R;
        const uint32_t* src = SQR || ONE ? sa : sb;
#pragma unroll 1
        for (int g = tid; g < Gr::G; g += T) {
            const Gr gr(g);
            uint32_t x[1 << R];
#pragma unroll
            for (int j = 0; j < (1 << R); ++j) x[j] = src[gr.at(j)];
            dif_regs<LAZY, R, Gr::HI, Gr::LO>(x, gr.base_low, twf, p);
            uint4 av{};
#pragma unroll
            for (int j = 0; j < (1 << R); ++j) {
                uint32_t o = x[j];
                if constexpr (ONE) {  // parked by this thread
                    if (j % 4 == 0) av = reinterpret_cast<const uint4*>(row_a + gr.base)[j / 4];
                    o = j % 4 == 0 ? av.x : j % 4 == 1 ? av.y : j % 4 == 2 ? av.z : av.w;
                } else if constexpr (!SQR) {
                    o = sa[gr.at(j)];
                }
                // below p for factors below p; below 2p for factors below 2p, 4p < 2^32
                const uint32_t z = mont(x[j], o, p, np);
                x[j] = LAZY ? z : csub(z, p);
            }
            dit_regs<LAZY, R, Gr::HI, Gr::LO>(x, gr.base_low, twi, p);
#pragma unroll
            for (int j = 0; j < (1 << R); ++j) sa[gr.at(j)] = x[j];
        }
    }
    __syncthreads();
    dit_rounds<LAZY, L1, 1, T, NR - 2, 1>(sa, twi, p, tid);
    using Gr = Group<L1, 1, 0>;
#pragma unroll 2
    for (int g = tid; g < Gr::G; g += T) {
        const Gr gr(g);
        uint32_t x[1 << R0];
#pragma unroll
        for (int j = 0; j < (1 << R0); ++j) x[j] = sa[gr.at(j)];
        dit_regs<LAZY, R0, Gr::HI, Gr::LO>(x, gr.base_low, twi, p);
        const uint2 bw = shoup_of(
            csub(mont(inter_twiddle(c, q, 1, (k2 * gr.base) & (uint32_t)(nn - 1), a.log_n, p), scale, p, np), p), p, np);
#pragma unroll
        for (int j = 0; j < (1 << R0); ++j) row_a[gr.idx(j)] = shoup2<LAZY>(x[j], sT[j], bw, p);
    }
    pdl_trigger();
}

// ---- 3: inverse columns ---------------------------------------------------------------

template <bool LAZY, int L2, int T>
__global__ void __launch_bounds__(T, wide_col_blocks(L2, false)) k_wide_inv(const WideArgs a) {
    using P2 = Plan<L2>;
    constexpr int NR = P2::nr;
    extern __shared__ __align__(16) uint32_t sm[];  // [2^L2][8]
    const NttConsts& c = c_wide[a.set];
    const int q = blockIdx.y;
    const uint32_t p = c.pr[q].p;
    const uint2* twi = c.stage[q][1];
    uint32_t* y = wide_planes(a, blockIdx.z) + ((size_t)q << a.log_n) + blockIdx.x * kWideCols;
    pdl_wait();
    {
        using Gr = Group<L2, kWideCols, NR - 1>;
        constexpr int R = Gr::R;
#pragma unroll 2
        for (int g = threadIdx.x; g < Gr::G; g += T) {
            const Gr gr(g);
            uint32_t x[1 << R];
#pragma unroll
            for (int j = 0; j < (1 << R); ++j) x[j] = y[((size_t)gr.idx(j) << a.log_n1) + gr.col];
            dit_regs<LAZY, R, Gr::HI, Gr::LO>(x, gr.base_low, twi, p);
#pragma unroll
            for (int j = 0; j < (1 << R); ++j) sm[gr.at(j)] = x[j];
        }
    }
    __syncthreads();
    dit_rounds<LAZY, L2, kWideCols, T, NR - 2, 1>(sm, twi, p, threadIdx.x);
    using Gr = Group<L2, kWideCols, 0>;
    constexpr int R = Gr::R;
#pragma unroll 2
    for (int g = threadIdx.x; g < Gr::G; g += T) {
        const Gr gr(g);
        uint32_t x[1 << R];
#pragma unroll
        for (int j = 0; j < (1 << R); ++j) x[j] = sm[gr.at(j)];
        dit_regs<LAZY, R, Gr::HI, Gr::LO>(x, gr.base_low, twi, p);
#pragma unroll
        for (int j = 0; j < (1 << R); ++j)
            y[((size_t)gr.idx(j) << a.log_n1) + gr.col] = Bfly<LAZY>::reduce(x[j], p);
    }
    pdl_trigger();
}

// ---- 1 to 3 of short transforms ------------------------------------------------------

// Threads of an operand.
__host__ __device__ constexpr int wide_short_threads(int l) { return l <= 9 ? 32 : 1 << (l - 4); }

// Up to 2^12 points: the whole product of one prime in one CTA, both operands'
// transforms at once in halves of the threads.  Loads, rounds and the
// pointwise product are those of the passes above; nothing goes through memory
// in between and there are no inter-pass twiddles.  us per product back to back,
// four launches -> two: 2^10 points 11.5 -> 6.7, 2^11 9.5 -> 8.5, 2^12 9.7 -> 11.1,
// but from the host, whose launches bound them, 14.2 -> 9.6 at 2^11 and no more at
// 2^12; three primes at 2^10 32-bit digits 11.3, here at 2^9 points 6.7.
// A batch: product tree of 2^20 leaves 2.28 -> 2.07 ms.
template <int L, int NP, bool SQR>
__global__ void __launch_bounds__(wide_short_threads(L) * (SQR ? 1 : 2)) k_wide_short(const WideFwdArgs fa) {
    constexpr int T = wide_short_threads(L), TT = SQR ? T : 2 * T;
    using P = Plan<L>;
    constexpr int NR = P::nr;
    static_assert(NR > 1, "several rounds");
    extern __shared__ __align__(16) uint32_t sm[];  // A's row, B's
    const NttConsts& c = c_wide[wide_set_index(NP, true)];
    const int q = blockIdx.x, op = SQR ? 0 : (int)threadIdx.x / T, tid = (int)threadIdx.x - op * T;
    const uint32_t product = blockIdx.z;
    const uint32_t p = c.pr[q].p, np = 0u - c.pr[q].pinv;
    const uint2* twf = c.stage[q][0];
    const uint2* twi = c.stage[q][1];
    const uint32_t scale = c_scale[wide_set_index(NP, true)][L][q];
    uint32_t* s = sm + ((uint32_t)op << L);
    pdl_wait();
    const OperandDesc in = wide_operand(fa, product, op);
    uint32_t* y = wide_planes(fa.w, product) + ((size_t)q << L);
    wide_load<true, L, 1, T, NP>(0, in, (size_t)1 << L, c, q, 0, s, tid);
    __syncthreads();
    dif_rounds<true, L, 1, T, 1, NR - 2>(s, twf, p, tid);
    if constexpr (!SQR) {
        smem_round<true, L, 1, T, NR - 1, false>(s, twf, p, tid);
        __syncthreads();
    }
    {  // the last DIF round of a square, the pointwise product, the first DIT round
        using Gr = Group<L, 1, NR - 1>;
        constexpr int R = Gr::R;
#pragma unroll 1
        for (int g = threadIdx.x; g < Gr::G; g += TT) {
            const Gr gr(g);
            uint32_t x[1 << R];
#pragma unroll
            for (int j = 0; j < (1 << R); ++j) x[j] = sm[gr.at(j)];
            if constexpr (SQR) dif_regs<true, R, Gr::HI, Gr::LO>(x, gr.base_low, twf, p);
#pragma unroll
            for (int j = 0; j < (1 << R); ++j) x[j] = mont(x[j], SQR ? x[j] : sm[(1u << L) + gr.at(j)], p, np);
            dit_regs<true, R, Gr::HI, Gr::LO>(x, gr.base_low, twi, p);
#pragma unroll
            for (int j = 0; j < (1 << R); ++j) sm[gr.at(j)] = x[j];
        }
    }
    __syncthreads();
    dit_rounds<true, L, 1, TT, NR - 2, 1>(sm, twi, p, threadIdx.x);
    using Gr = Group<L, 1, 0>;
    constexpr int R = Gr::R;
    const uint2 sc = shoup_of(scale, p, np);
#pragma unroll 1
    for (int g = threadIdx.x; g < Gr::G; g += TT) {
        const Gr gr(g);
        uint32_t x[1 << R];
#pragma unroll
        for (int j = 0; j < (1 << R); ++j) x[j] = sm[gr.at(j)];
        dit_regs<true, R, Gr::HI, Gr::LO>(x, gr.base_low, twi, p);
#pragma unroll
        for (int j = 0; j < (1 << R); ++j) y[gr.idx(j)] = csub(shoup_lazy(x[j], sc.x, sc.y, p), p);
    }
    pdl_trigger();
}

// ---- 4: CRT and carries --------------------------------------------------------------

// C += a b, 64 bits, with the carry out counted in k.
__device__ __forceinline__ void mac_count(uint32_t a, uint32_t b, uint32_t (&C)[2], uint32_t& k) {
    asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\t"
        "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
        "addc.u32 %2, %2, 0;"
        : "+r"(C[0]), "+r"(C[1]), "+r"(k)
        : "r"(a), "r"(b));
}
__device__ __forceinline__ void mac(uint32_t a, uint32_t b, uint32_t (&C)[2]) {
    asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\t"
        "madc.hi.u32 %1, %2, %3, %1;"
        : "+r"(C[0]), "+r"(C[1])
        : "r"(a), "r"(b));
}

// W += v on N words; the carry out is dropped.
template <int N>
__device__ __forceinline__ void add_words(uint32_t* W, const uint32_t* v) {
    static_assert(N >= 3, "add_words");
    if constexpr (N == 3)
        asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
            : "+r"(W[0]), "+r"(W[1]), "+r"(W[2])
            : "r"(v[0]), "r"(v[1]), "r"(v[2]));
    else if constexpr (N == 4)
        asm("add.cc.u32 %0, %0, %4;\n\taddc.cc.u32 %1, %1, %5;\n\taddc.cc.u32 %2, %2, %6;\n\taddc.u32 %3, %3, %7;"
            : "+r"(W[0]), "+r"(W[1]), "+r"(W[2]), "+r"(W[3])
            : "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]));
    else if constexpr (N == 5)
        asm("add.cc.u32 %0, %0, %5;\n\taddc.cc.u32 %1, %1, %6;\n\taddc.cc.u32 %2, %2, %7;\n\t"
            "addc.cc.u32 %3, %3, %8;\n\taddc.u32 %4, %4, %9;"
            : "+r"(W[0]), "+r"(W[1]), "+r"(W[2]), "+r"(W[3]), "+r"(W[4])
            : "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]));
    else if constexpr (N == 6)
        asm("add.cc.u32 %0, %0, %6;\n\taddc.cc.u32 %1, %1, %7;\n\taddc.cc.u32 %2, %2, %8;\n\t"
            "addc.cc.u32 %3, %3, %9;\n\taddc.cc.u32 %4, %4, %10;\n\taddc.u32 %5, %5, %11;"
            : "+r"(W[0]), "+r"(W[1]), "+r"(W[2]), "+r"(W[3]), "+r"(W[4]), "+r"(W[5])
            : "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]));
    else if constexpr (N == 7)
        asm("add.cc.u32 %0, %0, %7;\n\taddc.cc.u32 %1, %1, %8;\n\taddc.cc.u32 %2, %2, %9;\n\t"
            "addc.cc.u32 %3, %3, %10;\n\taddc.cc.u32 %4, %4, %11;\n\taddc.cc.u32 %5, %5, %12;\n\taddc.u32 %6, %6, %13;"
            : "+r"(W[0]), "+r"(W[1]), "+r"(W[2]), "+r"(W[3]), "+r"(W[4]), "+r"(W[5]), "+r"(W[6])
            : "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]));
    else {
        uint32_t cy = 0;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const uint64_t t = (uint64_t)W[k] + v[k] + cy;
            W[k] = (uint32_t)t;
            cy = (uint32_t)(t >> 32);
        }
    }
}

// Adds the coefficient with residues y (each below its p) to the words
// W[0 .. NP-1], the last taking the carry: sum y_i M/p_i - q M.  The NP products of
// a 32-bit limb of the M/p_i sum to a 64-bit column and a carry count (LAZY: the
// first four, p < 2^30, cannot overflow).  q = floor(sum y_i / p_i) in single
// precision from the top bits of y_i, put below an exponent byte: the float is
// 2^23 + floor(y_i / 256), and c.bias takes the 2^23 out again.  x / M is below
// 0.9 and the bias keeps 0.05 on either side, well above the rounding.  -q M
// comes from a table in shared memory (`nqm`, NP words a q): lanes with
// different q hit different banks there, a constant bank would serve them one
// by one (measured the constant bank: 29.5 us for the whole pass at 2^21 points, with the table 26.8).
template <bool LAZY, int NP>
__device__ __forceinline__ void add_crt(const WideCrt& c, const uint32_t* nqm, const uint32_t (&y)[NP], uint32_t* W) {
    float f = c.bias;
#pragma unroll
    for (int i = 0; i < NP; ++i) f = fmaf(__uint_as_float(__byte_perm(y[i], 0x4b000000u, 0x7321)), c.inv[i], f);
    const uint32_t* s = nqm + NP * min((int)f, NP - 1);
    uint32_t lo[NP], hi[NP], k[NP] = {};  // columns and their carry counts
#pragma unroll
    for (int l = 0; l < NP - 1; ++l) {
        const uint64_t t = (uint64_t)y[0] * c.m[0][l];
        uint32_t C[2] = {(uint32_t)t, (uint32_t)(t >> 32)};
#pragma unroll
        for (int i = 1; i < NP; ++i) {
            if (LAZY && i < 4)
                mac(y[i], c.m[i][l], C);
            else
                mac_count(y[i], c.m[i][l], C, k[l]);
        }
        lo[l] = C[0], hi[l] = C[1];
    }
    lo[NP - 1] = k[NP - 3];  // word l + 2 takes column l's count; the sum is mod 2^(32 NP)
    k[NP - 3] = 0;
    add_words<NP>(W, lo);
    add_words<NP - 1>(W + 1, hi);
    add_words<NP - 2>(W + 2, k);
    uint32_t m[NP];
#pragma unroll
    for (int l = 0; l < NP; ++l) m[l] = s[l];
    add_words<NP>(W, m);
}

__device__ __forceinline__ uint64_t add_c(uint64_t a, uint64_t b, uint32_t& cy) {
    const uint64_t t = a + b, r = t + cy;
    cy = (uint32_t)(t < a) + (uint32_t)(r < t);
    return r;
}

// Chunk c (coefficients 4c .. 4c+3): their exact sum as the chunk's NP - 1 limbs D
// and a spill of two limbs (below 2^122: a coefficient is below 2^(2 D + 22) for
// digits of D <= 96 bits).
template <bool LAZY, int NP>
__device__ __forceinline__ void chunk_sum(const WideCrt& crt, const uint32_t* nqm, const uint32_t* y, size_t nn,
                                          size_t c, uint64_t (&D)[NP - 1], uint64_t (&sp)[2]) {
    uint32_t r[4][NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const uint4 v = *reinterpret_cast<const uint4*>(y + i * nn + 4 * c);
        r[0][i] = v.x, r[1][i] = v.y, r[2][i] = v.z, r[3][i] = v.w;
    }
    // A coefficient is added where the words above the sum so far are still
    // zero, and the sum so far leaves room in its NP words.
    uint32_t W[2 * (NP + 1)] = {};
    if constexpr (NP == 6) {  // 80-bit digits: the odd ones start in the middle of a word
        uint32_t O[11] = {};
        add_crt<LAZY, NP>(crt, nqm, r[0], W);
        add_crt<LAZY, NP>(crt, nqm, r[2], W + 5);
        add_crt<LAZY, NP>(crt, nqm, r[1], O);
        add_crt<LAZY, NP>(crt, nqm, r[3], O + 5);
        uint32_t V[12];
        V[0] = O[0] << 16;
#pragma unroll
        for (int k = 1; k < 11; ++k) V[k] = __funnelshift_l(O[k - 1], O[k], 16);
        V[11] = O[10] >> 16;
        add_words<12>(W + 2, V);
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) add_crt<LAZY, NP>(crt, nqm, r[k], W + k * (int)(wide_bits(NP) / 32));
    }
#pragma unroll
    for (int k = 0; k < NP - 1; ++k) D[k] = W[2 * k] | ((uint64_t)W[2 * k + 1] << 32);
    sp[0] = W[2 * NP - 2] | ((uint64_t)W[2 * NP - 1] << 32);
    sp[1] = W[2 * NP] | ((uint64_t)W[2 * NP + 1] << 32);
}

// The 28-bit digits that start in chunk c, whose final limbs are S; the last
// one may reach into the final low limb `next` of the chunk above.
template <int NL>
__device__ __forceinline__ void store_digits28(uint32_t* o, size_t out_cap, uint64_t c, const uint64_t (&S)[NL],
                                               uint64_t next) {
    constexpr uint32_t kBits = 64 * NL;
    const uint64_t mask = (1u << 28) - 1u;
    const uint64_t bit0 = c * kBits;
    uint64_t k = (bit0 + 27) / 28;
    const uint64_t kend = min((bit0 + kBits + 27) / 28, (uint64_t)out_cap);
    const uint32_t off0 = (uint32_t)(k * 28 - bit0);  // < 28
    uint64_t cur = S[0] >> off0;
    int have = 64 - (int)off0;
#pragma unroll
    for (int w = 1; w <= NL; ++w) {
        const uint64_t nxtw = w < NL ? S[w % NL] : next;
        while (have >= 28) {
            if (k < kend) o[k] = (uint32_t)(cur & mask);
            ++k;
            cur >>= 28;
            have -= 28;
        }
        if (k < kend) o[k] = (uint32_t)((cur | (nxtw << have)) & mask);
        ++k;
        cur = nxtw >> (28 - have);
        have = 36 + have;
    }
}

// One chunk of NP - 1 limbs a thread, 256 chunks a block; a ninth warp recomputes the
// 32 chunks below the block, whose carries almost always settle the block's
// carry-in without waiting for another block (else the decoupled look-back on
// the blocks' flags, in ticket order).  Chunk c's value is
// (D_c + spill_{c-1} + carry_c) mod 2^(64 (NP - 1)) with one-bit carries.
constexpr int kWideCarryWarps = kWideCarryChunks / 32;
template <bool LAZY, int NP>
__global__ void __launch_bounds__(kWideCarryChunks + 32) k_wide_carry(const __grid_constant__ WideCarryArgs a) {
    constexpr int NL = NP - 1;
    const WideCrt& crt = c_crt[wide_set_index(NP, LAZY)];
    __shared__ uint32_t s_bid, s_cin, s_win_g, s_win_p;
    __shared__ uint32_t s_wg[kWideCarryWarps], s_wp[kWideCarryWarps];
    __shared__ uint64_t s_sp[kWideCarryWarps + 1][2];
    __shared__ uint64_t s_low[kWideCarryChunks];  // 28-bit output: each chunk's low limb before its spill and carry
    __shared__ uint32_t s_nqm[NP * NP];
    if (threadIdx.x == 0) s_bid = (uint32_t)(atomicAdd(a.ticket, 1ull) - a.ticket_base);
    for (int i = threadIdx.x; i < NP * NP; i += kWideCarryChunks + 32) s_nqm[i] = crt.nqm[i / NP][i % NP];
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    if (s_bid >= gridDim.x) {  // the ticket counter and the launch disagree: report, touch nothing
        if (threadIdx.x == 0) atomicOr(a.err, 2u);
        return;
    }
    const uint32_t bid = s_bid % a.bpp;
    const uint32_t product = s_bid / a.bpp;
    ProductDesc pd;
    if (a.descs) {
        pd = a.descs[product];
    } else {
        pd.y = a.y + (((size_t)product * (uint32_t)(a.nops * NP)) << a.log_n);
        pd.flags = a.flags + (size_t)product * a.bpp;
        pd.out = static_cast<char*>(a.out) + (int64_t)product * a.step_out;
        pd.out_cap = a.out_cap;
    }
    // a product of a batch shorter than its class's longest: no later block waits on these
    if (bid >= wide_carry_blocks(NP, pd.out_cap, a.out_fmt)) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool window = warp == kWideCarryWarps;
    const size_t nn = (size_t)1 << a.log_n;
    const uint32_t nch = (uint32_t)(nn / 4);
    const int64_t c = (int64_t)bid * kWideCarryChunks + (window ? lane - 32 : (int)threadIdx.x);
    uint64_t S[NL] = {}, sp[2] = {0, 0};
    if (c >= 0 && c < nch) chunk_sum<LAZY, NP>(crt, s_nqm, pd.y, nn, (size_t)c, S, sp);
    if (!window) s_low[threadIdx.x] = S[0];
    if (lane == 31) {
        s_sp[warp][0] = sp[0];
        s_sp[warp][1] = sp[1];
    }
    uint64_t p0 = __shfl_up_sync(0xffffffffu, sp[0], 1), p1 = __shfl_up_sync(0xffffffffu, sp[1], 1);
    __syncthreads();
    if (lane == 0) {
        p0 = window ? 0 : s_sp[warp ? warp - 1 : kWideCarryWarps][0];
        p1 = window ? 0 : s_sp[warp ? warp - 1 : kWideCarryWarps][1];
    }
    uint32_t g = 0;
    S[0] = add_c(S[0], p0, g);
    S[1] = add_c(S[1], p1, g);
    uint64_t all = S[0] & S[1];
#pragma unroll
    for (int k = 2; k < NL; ++k) {
        S[k] = add_c(S[k], 0, g);
        all &= S[k];
    }
    const uint32_t pbit = all == ~0ull;
    // the window's lowest chunk lacks its predecessor's spill: it neither
    // stops nor makes a carry there, except below chunk 0
    const uint32_t gm = __ballot_sync(0xffffffffu, g);
    uint32_t pm = __ballot_sync(0xffffffffu, pbit);
    if (window && bid != 0) pm |= 1u;
    const uint32_t bm = gm | pm;
    if (lane == 0) {
        if (window) {
            s_win_g = gm;
            s_win_p = pm;
        } else {
            s_wg[warp] = (uint32_t)((((uint64_t)gm + bm) >> 32) & 1u);
            s_wp[warp] = pm == 0xffffffffu;
        }
    }
    __syncthreads();
    // The block's flag holds all that a later block reads, so its stores need
    // no ordering; the inclusive one comes after the barrier that releases the
    // block's own threads.
    uint32_t bG = 0, bP = 1, cin = 0;
    if (threadIdx.x == 0) {
        for (int w = 0; w < kWideCarryWarps; ++w) {
            bG = s_wg[w] | (s_wp[w] & bG);
            bP = bP & s_wp[w];
        }
        const uint32_t stop = ~s_win_p;  // window chunks that do not propagate a carry
        if (bid == 0) {
            bP = 0;
        } else if (stop) {
            cin = (s_win_g >> (31 - __clz(stop))) & 1u;
        } else {
            uint64_t* flags = pd.flags;
            cuda::atomic_ref<unsigned long long, cuda::thread_scope_device>(
                *reinterpret_cast<unsigned long long*>(flags + bid))
                .store(make_flag(a.epoch, 1, bG, bP), cuda::memory_order_relaxed);
            for (int k = (int)bid - 1;; --k) {  // block 0 is inclusive
                const uint64_t f = wait_flag(flags + k, a.epoch, kSpinLimit, a.err);
                if (f == 0) break;  // gave up: error recorded, carry taken as 0
                const uint32_t st = (uint32_t)(f >> 2) & 3u, fg = (uint32_t)(f >> 1) & 1u, fp = (uint32_t)f & 1u;
                if (st == 2 || fg || !fp) {
                    cin = fg;
                    break;
                }
            }
        }
        s_cin = cin;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        cuda::atomic_ref<unsigned long long, cuda::thread_scope_device>(
            *reinterpret_cast<unsigned long long*>(pd.flags + bid))
            .store(make_flag(a.epoch, 2, bG | (bP & cin), 0), cuda::memory_order_relaxed);
    if (window) return;
    uint32_t cw = s_cin;
    for (int w = 0; w < warp; ++w) cw = s_wg[w] | (s_wp[w] & cw);
    const uint64_t sum = (uint64_t)gm + bm + cw;
    const uint32_t carries = (uint32_t)sum ^ gm ^ bm;
    uint32_t cy = (carries >> lane) & 1u;
#pragma unroll
    for (int k = 0; k < NL; ++k) {
        const uint64_t t = S[k] + cy;
        cy = cy & (t == 0);
        S[k] = t;
    }
    if (a.out_fmt == kFmtLimb64) {
        uint64_t* o = static_cast<uint64_t*>(pd.out);
        const size_t at = (size_t)c * NL;
        if (NL % 2 == 0 && at + NL <= pd.out_cap && (reinterpret_cast<uintptr_t>(o) & 15u) == 0) {
            ulonglong2* d = reinterpret_cast<ulonglong2*>(o + at);
#pragma unroll
            for (int k = 0; k + 1 < NL; k += 2) d[k / 2] = make_ulonglong2(S[k], S[k + 1]);
        } else {
#pragma unroll
            for (int k = 0; k < NL; ++k)
                if (at + k < pd.out_cap) o[at + k] = S[k];
        }
    } else {
        uint64_t next = 0;  // low limb of the next chunk: its raw sum, this chunk's spill and carry out
        if (threadIdx.x + 1 < kWideCarryChunks) {
            next = s_low[threadIdx.x + 1];
        } else if (c + 1 < nch) {
            uint32_t r[NP], w[NP] = {};
#pragma unroll
            for (int i = 0; i < NP; ++i) r[i] = pd.y[i * nn + 4 * (size_t)(c + 1)];
            add_crt<LAZY, NP>(crt, s_nqm, r, w);
            next = w[0] | ((uint64_t)w[1] << 32);
        }
        next += sp[0] + (lane == 31 ? (uint32_t)(sum >> 32) & 1u : (carries >> (lane + 1)) & 1u);
        store_digits28<NL>(static_cast<uint32_t*>(pd.out), pd.out_cap, (uint64_t)c, S, next);
    }
}

// ---- launches ------------------------------------------------------------------------

namespace {

template <bool LAZY, int L2, int NP>
cudaError_t launch_fwd(const WideFwdArgs& fa, uint32_t count, cudaStream_t st) {
    constexpr int RL = Plan<L2>::r(Plan<L2>::nr - 1);
    const size_t sm = ((size_t)kWideCols * 4 << L2) + kWideCols * ((1 << RL) + 1) * sizeof(uint2);
    auto k = k_wide_fwd<LAZY, L2, wide_col_threads(L2, true), NP>;
    allow_smem(k, sm);
    return launch_k(k, dim3((1u << fa.w.log_n1) / kWideCols, NP, count * fa.w.nops), dim3(wide_col_threads(L2, true)), sm,
                    st, fa);
}
template <bool LAZY, int L2>
cudaError_t launch_cols(bool fwd, const WideFwdArgs& fa, uint32_t count, cudaStream_t st) {
    const WideArgs& a = fa.w;
    if (fwd)
        return a.np == 5   ? launch_fwd<LAZY, L2, 5>(fa, count, st)
               : a.np == 6 ? launch_fwd<LAZY, L2, 6>(fa, count, st)
                           : launch_fwd<LAZY, L2, 7>(fa, count, st);
    const size_t tile = (size_t)kWideCols * 4 << L2;
    auto k = k_wide_inv<LAZY, L2, wide_col_threads(L2, false)>;
    allow_smem(k, tile);
    return launch_k(k, dim3((1u << a.log_n1) / kWideCols, a.np, count), dim3(wide_col_threads(L2, false)), tile, st, a);
}

template <bool LAZY>
cudaError_t dispatch_cols(int l2, bool fwd, const WideFwdArgs& a, uint32_t count, cudaStream_t st) {
    switch (l2) {
        case 5: return launch_cols<LAZY, 5>(fwd, a, count, st);
        case 6: return launch_cols<LAZY, 6>(fwd, a, count, st);
        case 7: return launch_cols<LAZY, 7>(fwd, a, count, st);
        case 8: return launch_cols<LAZY, 8>(fwd, a, count, st);
        case 9: return launch_cols<LAZY, 9>(fwd, a, count, st);
        case 10: return launch_cols<LAZY, 10>(fwd, a, count, st);
        case 11: return launch_cols<LAZY, 11>(fwd, a, count, st);
        default: return cudaErrorInvalidValue;
    }
}

template <bool LAZY, int L1, bool SQR>
cudaError_t launch_rows_of(const WideArgs& a, uint32_t count, cudaStream_t st) {
    static_assert(L1 <= kMaxLogWideRow, "stage tables");
    constexpr int RP = wide_rows_per_cta(L1);
    const size_t sm = (size_t)RP * wide_row_words(L1, SQR) * 4;
    auto k = k_wide_rows<LAZY, L1, SQR>;
    allow_smem(k, sm);
    return launch_k(k, dim3((1u << (a.log_n - L1)) / RP, a.np, count), dim3(wide_row_threads(L1) * RP), sm, st, a);
}
template <bool LAZY, int L1>
cudaError_t launch_rows(const WideArgs& a, bool square, uint32_t count, cudaStream_t st) {
    return square ? launch_rows_of<LAZY, L1, true>(a, count, st) : launch_rows_of<LAZY, L1, false>(a, count, st);
}

template <bool LAZY>
cudaError_t dispatch_rows(int l1, const WideArgs& a, bool square, uint32_t count, cudaStream_t st) {
    switch (l1) {
        case 5: return launch_rows<LAZY, 5>(a, square, count, st);
        case 6: return launch_rows<LAZY, 6>(a, square, count, st);
        case 7: return launch_rows<LAZY, 7>(a, square, count, st);
        case 8: return launch_rows<LAZY, 8>(a, square, count, st);
        case 9: return launch_rows<LAZY, 9>(a, square, count, st);
        case 10: return launch_rows<LAZY, 10>(a, square, count, st);
        case 11: return launch_rows<LAZY, 11>(a, square, count, st);
        case 12: return launch_rows<LAZY, 12>(a, square, count, st);
        case 13: return launch_rows<LAZY, 13>(a, square, count, st);
        case 14: return launch_rows<LAZY, 14>(a, square, count, st);
        default: return cudaErrorInvalidValue;
    }
}

WideCrt make_crt(const PrimeSetInfo& ps) {
    WideCrt c{};
    const int np = ps.np;
    double off = 0;
    using Words = uint32_t[kWideMaxPrimes];
    auto times = [np](Words& x, uint32_t v) {
        uint64_t cy = 0;
        for (int k = 0; k < np; ++k) {
            cy += (uint64_t)x[k] * v;
            x[k] = (uint32_t)cy;
            cy >>= 32;
        }
    };
    Words M = {1};
    for (int i = 0; i < np; ++i) {
        Words x = {1};
        for (int j = 0; j < np; ++j)
            if (j != i) times(x, ps.p[j]);
        std::memcpy(c.m[i], x, sizeof(c.m[i]));
        times(M, ps.p[i]);
        c.inv[i] = (float)(256.0 / ps.p[i]);
        off += 8388608.0 * (double)c.inv[i];
    }
    c.bias = (float)(0.05 - off);
    for (int q = 0; q < np; ++q) {
        Words x;
        std::memcpy(x, M, sizeof(x));
        times(x, (uint32_t)q);
        uint64_t cy = 1;  // its negative
        for (int k = 0; k < np; ++k) {
            cy += (uint32_t)~x[k];
            c.nqm[q][k] = (uint32_t)cy;
            cy >>= 32;
        }
    }
    return c;
}

uint32_t pow_m(uint64_t b, uint32_t e, uint32_t p) {
    uint64_t r = 1;
    for (b %= p; e; e >>= 1, b = b * b % p)
        if (e & 1) r = r * b % p;
    return (uint32_t)r;
}

template <int L, int NP>
cudaError_t launch_short_of(const WideFwdArgs& fa, uint32_t count, cudaStream_t st) {
    const size_t sm = (size_t)4 * fa.w.nops << L;
    const dim3 grid(NP, 1, count);
    return fa.w.nops == 1 ? launch_k(k_wide_short<L, NP, true>, grid, dim3(wide_short_threads(L)), sm, st, fa)
                          : launch_k(k_wide_short<L, NP, false>, grid, dim3(2 * wide_short_threads(L)), sm, st, fa);
}
template <int L>
cudaError_t launch_short(const WideFwdArgs& fa, uint32_t count, cudaStream_t st) {
    return fa.w.np == 5   ? launch_short_of<L, 5>(fa, count, st)
           : fa.w.np == 6 ? launch_short_of<L, 6>(fa, count, st)
                          : launch_short_of<L, 7>(fa, count, st);
}
cudaError_t dispatch_short(const WideFwdArgs& fa, uint32_t count, cudaStream_t st) {
    switch (fa.w.log_n) {
        case 8: return launch_short<8>(fa, count, st);
        case 9: return launch_short<9>(fa, count, st);
        case 10: return launch_short<10>(fa, count, st);
        case 11: return launch_short<11>(fa, count, st);
        case 12: return launch_short<12>(fa, count, st);
        default: return cudaErrorInvalidValue;
    }
}

// 1 / N / (M / p) mod p times a power of two, Montgomery form: the inverse
// transform's 1/N, the CRT's (M/p)^-1, and 2^32 for the pointwise product and
// each reduction of the two digits (one each, two for three words).
void set_scale(const PrimeSetInfo& ps, int log_n, uint32_t* scale) {
    for (int i = 0; i < ps.np; ++i) {
        const uint32_t p = ps.p[i];
        uint64_t d = pow_m(2, (uint32_t)log_n, p);
        for (int j = 0; j < ps.np; ++j)
            if (j != i) d = d * (ps.p[j] % p) % p;
        const uint64_t v = (uint64_t)pow_m(d, p - 2, p) * pow_m(2, ps.np == 5 ? 96 : 160, p) % p;
        scale[i] = (uint32_t)((v << 32) % p);
    }
}

}  // namespace

cudaError_t upload_wide_consts(int set, const NttConsts& c) {
    const int w = set - kFirstWideSet;
    const PrimeSetInfo& ps = kPrimeSets[set];
    const WideCrt crt = make_crt(ps);
    uint32_t scale[kWideMaxLogN + 1][kWideMaxPrimes] = {};
    for (int ln = kWideMinLogN; ln <= ps.log_max; ++ln) set_scale(ps, ln, scale[ln]);
    cudaError_t e = cudaMemcpyToSymbol(c_crt, &crt, sizeof(crt), w * sizeof(crt));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_scale, scale, sizeof(scale), w * sizeof(scale));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_wide, &c, sizeof(NttConsts), w * sizeof(NttConsts));
    return e;
}

// Built-in column lengths, the fastest measured on B200 for one product and
// for a batch that fills the GPU (two operands of half the points).  us per
// product back to back, the choice against the nearest other length: 2^17 points 21.0 (2^6) / 22.2 (2^7), 2^18 28.9 (2^8) /
// 29.8 (2^7), 2^19 47.7 (2^8) / 49.5 (2^9), 2^20 88.7 (2^8) / 90.4 (2^9), 2^21 175.7
// (2^10) / 180.5 (2^9), 2^23 753 (2^10) / 780 (2^11), 2^24 1543 (2^10) / 1572 (2^11).
// Batches, us per 2^19 points: 2^13 33.7 (2^7) / 35.7 (2^6), 2^15 34.5 (2^8) /
// 35.4 (2^7), 2^17 37.8 (2^9) / 38.8 (2^8), 2^19 38.7 (2^8) / 40.4 (2^9).
static constexpr int8_t kWideColumn[kWideMaxLogN + 1] = {0, 0, 0, 0, 0, 0, 0, 0, 0,  0,  0,  0,  0,
                                                         7, 8, 8, 8, 6, 8, 8, 8, 10, 10, 10, 10, 11};
static constexpr int8_t kWideBatchColumn[kWideMaxLogN + 1] = {0, 0, 0, 0, 0, 0, 0, 0, 0,  0,  0,  0,  0,
                                                              7, 8, 8, 8, 9, 8, 8, 9, 10, 10, 10, 10, 11};

TransformShape wide_shape(int log_n, bool batch) {
    TransformShape s{log_n, 0, 0};
    if (log_n <= kWideShortMaxLogN || log_n > kWideMaxLogN) return s;
    auto built = [&](int l2) { return l2 >= 5 && l2 <= 11 && log_n - l2 >= 5 && log_n - l2 <= 14; };
    const int tuned = tuned_split(log_n + 1, batch);
    s.log_n2 = built(tuned) ? tuned : (batch ? kWideBatchColumn : kWideColumn)[log_n];
    s.log_n1 = log_n - s.log_n2;
    return s;
}

const char* const kWideKernelNames[2][kNttLaunches] = {{"k_wide_fwd", "k_wide_rows", "k_wide_inv", "k_wide_carry"},
                                                       {"k_wide_short", "none", "none", "k_wide_carry"}};

// Longest transform over np primes.
static int wide_max_log(int np) { return kPrimeSets[kFirstWideSet + 2 * (np - kWidePrimes) + 1].log_max; }

// The shortest transform that holds the product, over the fewest primes that
// reach it: at the same length six primes cost 1.25 times as much as five and
// seven 1.4 (1.4 and 1.6 where only they need the strict set), twice the points
// of five 1.8 to 2.  us per product at the longest operands of each form:
// 2^18 points over six 36, over seven 40, 2^19 over five 48; 2^19 over six 60, over seven 71,
// 2^20 over five 88; 2^22 over six 488, over seven 561, 2^23 over five 755.
WideForm wide_form(uint32_t nd32a, uint32_t nd32b, int min_long) {
    WideForm best;
    for (int np = kWidePrimes; np <= kWideMaxPrimes; ++np) {
        const uint64_t points = (uint64_t)wide_digits(np, nd32a) + wide_digits(np, nd32b) - 1;
        int ln = kWideMinLogN - 1;
        while (ln <= kWideMaxLogN && ((uint64_t)1 << ln) < points) ++ln;
        if (ln < (np == kWidePrimes ? kWideMinLogN : min_long) || ln > wide_max_log(np)) continue;
        if (!best.np || ln < best.log_n) best = {np, ln};
    }
    return best;
}

cudaError_t launch_wide_product(WideForm f, const ProductDesc* descs, const ProductDesc& one, const WideStep& step,
                                uint32_t count, bool square, int out_fmt, uint32_t bpp, const CarryLaunch& cl, cudaStream_t st,
                                cudaEvent_t* ev) {
    const int log_n = f.log_n;
    if (f.np < kWidePrimes || f.np > kWideMaxPrimes || log_n > wide_max_log(f.np) || count < 1 || count > kBatchPiece)
        return cudaErrorInvalidValue;
    const bool whole = log_n <= kWideShortMaxLogN;
    const int l2 = wide_shape(log_n, descs != nullptr || count > 1).log_n2;
    if (log_n < kWideMinLogN || (!whole && !l2)) return cudaErrorInvalidValue;
    const int w = wide_set_for(f.np, log_n) - kFirstWideSet;
    const bool lazy = w % 2 == 0;
    WideFwdArgs fa{};
    WideArgs& a = fa.w;
    a.descs = descs;
    a.y = one.y;
    a.nops = square ? 1 : 2;
    a.log_n = log_n;
    a.log_n1 = log_n - l2;
    a.np = f.np;
    a.set = w;
    fa.op[0] = one.op[0];
    fa.op[1] = one.op[1];
    fa.step_a = step.a;
    fa.step_b = step.b;
    if (ev) cudaEventRecord(ev[0], st);
    cudaError_t e = cudaSuccess;
    if (whole) {
        e = dispatch_short(fa, count, st);
        if (ev) cudaEventRecord(ev[1], st);
        if (ev) cudaEventRecord(ev[2], st);
    } else {
        e = lazy ? dispatch_cols<true>(l2, true, fa, count, st) : dispatch_cols<false>(l2, true, fa, count, st);
        if (e != cudaSuccess) return e;
        if (ev) cudaEventRecord(ev[1], st);
        e = lazy ? dispatch_rows<true>(a.log_n1, a, square, count, st)
                 : dispatch_rows<false>(a.log_n1, a, square, count, st);
        if (e != cudaSuccess) return e;
        if (ev) cudaEventRecord(ev[2], st);
        e = lazy ? dispatch_cols<true>(l2, false, fa, count, st) : dispatch_cols<false>(l2, false, fa, count, st);
    }
    if (e != cudaSuccess) return e;
    if (ev) cudaEventRecord(ev[3], st);
    WideCarryArgs ca{};
    ca.descs = descs;
    ca.y = one.y;
    ca.flags = one.flags;
    ca.out = one.out;
    ca.out_cap = one.out_cap;
    ca.step_out = step.out;
    ca.nops = a.nops;
    ca.log_n = log_n;
    ca.out_fmt = out_fmt;
    ca.bpp = bpp;
    ca.ticket = cl.ticket;
    ca.ticket_base = cl.ticket_base;
    ca.epoch = cl.epoch;
    ca.err = cl.err;
    auto k = f.np == 5   ? (lazy ? k_wide_carry<true, 5> : k_wide_carry<false, 5>)
             : f.np == 6 ? (lazy ? k_wide_carry<true, 6> : k_wide_carry<false, 6>)
                         : (lazy ? k_wide_carry<true, 7> : k_wide_carry<false, 7>);
    e = launch_k(k, dim3(bpp * count), dim3(kWideCarryChunks + 32), 0, st, ca);
    if (ev) cudaEventRecord(ev[4], st);
    return e;
}

cudaError_t launch_wide_batch(WideForm f, const ProductDesc* descs, uint32_t count, bool square, int out_fmt,
                              uint32_t bpp, const CarryLaunch& cl, cudaStream_t st) {
    for (uint32_t done = 0; done < count; done += kBatchPiece) {
        CarryLaunch piece = cl;
        piece.ticket_base = cl.ticket_base + (uint64_t)done * bpp;
        const uint32_t n = count - done < kBatchPiece ? count - done : kBatchPiece;
        const cudaError_t e = launch_wide_product(f, descs + done, ProductDesc{}, WideStep{}, n, square, out_fmt,
                                                  bpp, piece, st, nullptr);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace bgpu
