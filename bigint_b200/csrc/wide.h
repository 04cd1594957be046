// The wide-digit product pipeline (wide_kernels.cu): 64-bit digits over five
// primes, 80-bit digits over six or 96-bit digits over seven.  Against 32-bit
// digits over three primes a product in 64-bit digits takes half the points
// with 5/3 of the residues each, 5/6 of the residues in all, and one transform
// level less; the longer digits fill the steps between powers of two.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "engine.h"

namespace bgpu {

// Bits of a digit over np primes, and the digits of nd32 32-bit digits.
__host__ __device__ constexpr uint32_t wide_bits(int np) { return 16u * (uint32_t)(np - 1); }
__host__ __device__ constexpr uint32_t wide_digits(int np, uint32_t nd32) {
    return (uint32_t)(((uint64_t)nd32 * 32 + wide_bits(np) - 1) / wide_bits(np));
}

constexpr int kWideMaxPrimes = 7;

// A single product takes more than five primes from here: below 2^16 points the
// launches' latencies count and the three-word digits load and reduce more
// slowly: us per product, 2^13 points over six primes 13.6, 2^14 over five 11.8;
// 2^15 over six 16.6, 2^16 over five 16.4; 2^16 over six 19.0, over seven 19.4, 2^17 over five 21.3.
constexpr int kLongDigitMinLogN = 16;

// Levels of equal products (product trees, decimal conversions) leave the
// schoolbook and Karatsuba kernels here, whatever their crossovers: us per 1024
// products, 192 limbs schoolbook 24.9, this 31.0; 256 limbs 37.0, Karatsuba
// 45.5, this 31.0; 512 limbs Karatsuba 115, this 31.
constexpr size_t kLevelSmallMaxLimbs = 192;

// Transform of a product: 2^log_n points over np primes (np == 0: none).
struct WideForm {
    int np = 0, log_n = 0;
};
// The form of least work for operands of nd32a and nd32b 32-bit digits; more
// than five primes from 2^min_long points.
WideForm wide_form(uint32_t nd32a, uint32_t nd32b, int min_long);

// Shortest transform, and the longest that one block does whole.
constexpr int kWideMinLogN = 8;
constexpr int kWideShortMaxLogN = 12;

// Products of one set of launches: descs, or one product moved by equal steps
// (bytes; planes and flags follow one another).  Launch arguments are kept
// short, the constants are in constant memory: the host's launches bound small
// products (2^11 points 14.8 us a call, with the CRT's constants and a full
// description of each product in the arguments 15.5).
struct WideArgs {              // column and row passes
    const ProductDesc* descs;  // y: nops * np planes of N residues (the result replaces A's)
    uint32_t* y;
    int nops, log_n, log_n1, np;
    int set;  // of the wide sets
};
struct WideFwdArgs {
    WideArgs w;
    OperandDesc op[2];
    int64_t step_a, step_b;
};

struct WideCarryArgs {
    const ProductDesc* descs;  // y, flags, out, out_cap
    uint32_t* y;
    uint64_t* flags;
    void* out;
    size_t out_cap;
    int64_t step_out;
    unsigned long long* ticket;
    uint64_t ticket_base, epoch;
    uint32_t* err;
    int nops, log_n, out_fmt;
    uint32_t bpp;  // blocks per product
};

// CRT of residues y_i = x (M/p_i)^-1 mod p_i: x = sum y_i M/p_i - q M, q < np.
struct WideCrt {
    uint32_t m[kWideMaxPrimes][kWideMaxPrimes - 1];  // M / p_i, np - 1 words
    uint32_t nqm[kWideMaxPrimes][kWideMaxPrimes];    // -q M mod 2^(32 np)
    float inv[kWideMaxPrimes];                       // 256 / p_i
    float bias;                                      // 0.05 - 2^23 sum inv
};

struct WideStep {
    int64_t a = 0, b = 0, out = 0;
};

constexpr uint32_t kWideCarryChunks = 256;  // chunks of four digits (np - 1 limbs) per carry block
// Carry blocks of a product with out_cap output elements.
__host__ __device__ inline uint32_t wide_carry_blocks(int np, size_t out_cap, int out_fmt) {
    const uint64_t limbs = out_fmt == kFmtLimb64 ? out_cap : ((uint64_t)out_cap * 28 + 63) / 64;
    const uint32_t per = (uint32_t)(np - 1) * kWideCarryChunks;
    return (uint32_t)((limbs + per - 1) / per);
}

// Split of 2^log_n points: the tuned one of 2^(log_n + 1) 32-bit digits
// (bgpu_set_split, bgpu_set_batch_split) where its kernels are built, else the
// built-in one.  log_n2 == 0: one block does it whole, or no transform of this length.
TransformShape wide_shape(int log_n, bool batch);
cudaError_t upload_wide_consts(int set, const NttConsts& c);
// Kernels of a form: four, or two where one block does a transform whole (the
// middle entries of its timing are empty).
inline uint32_t wide_launches(WideForm f) { return f.log_n <= kWideShortMaxLogN ? 2 : kNttLaunches; }
extern const char* const kWideKernelNames[2][kNttLaunches];

// The four launches of `count` products of one form (digits of both operands
// together at most 2^log_n + 1); each product's carry scan has `bpp` blocks
// (tickets).  At most kBatchPiece products.
cudaError_t launch_wide_product(WideForm f, const ProductDesc* descs, const ProductDesc& one, const WideStep& step,
                                uint32_t count, bool square, int out_fmt, uint32_t bpp,
                                const CarryLaunch& cl, cudaStream_t st, cudaEvent_t* ev);

// The same for any number of products in the device array `descs`, in pieces
// that fit a launch grid, all on one ticket sequence from cl.ticket_base.
cudaError_t launch_wide_batch(WideForm f, const ProductDesc* descs, uint32_t count, bool square, int out_fmt,
                              uint32_t bpp, const CarryLaunch& cl, cudaStream_t st);

}  // namespace bgpu
