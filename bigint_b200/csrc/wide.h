// The five-prime product pipeline: 64-bit digits over five primes
// (wide_kernels.cu).  Against 32-bit digits over three primes a product takes
// half the points with 5/3 of the residues each, 5/6 of the residues in all,
// and one transform level less.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "engine.h"

namespace bgpu {

// 64-bit digits of an operand.
__host__ __device__ inline uint32_t wide_digits(const OperandDesc& o) { return o.nd32 / 2 + o.nd32 % 2; }

// Shortest transform: below it (1024 limbs of product) the three-prime
// kernels, whose few blocks are as fast.
constexpr int kWideMinLogN = 10;

struct WideArgs {
    const ProductDesc* descs;  // y: (square ? 1 : 2) * 5 planes of N residues (the result replaces A's)
    ProductDesc one;
    int nops, log_n, log_n1;
    uint32_t scale[kWidePrimes];  // row pass: 2^96 / N / (M / p) mod p, Montgomery form
};

// CRT of five residues y_i = x (M/p_i)^-1 mod p_i: x = sum y_i M/p_i - q M.
constexpr int kWideMaxQ = 5;  // q is at most 4
struct WideCrt {
    uint32_t m[kWidePrimes][4];  // M / p_i
    uint32_t nqm[kWideMaxQ][5];  // -q M mod 2^160
    float inv[kWidePrimes];      // 256 / p_i
    float bias;                  // 0.05 - 2^23 sum inv
};

struct WideCarryArgs {
    const ProductDesc* descs;  // y, flags, out, out_cap
    ProductDesc one;
    WideCrt crt;
    int log_n, out_fmt;
    uint32_t bpp;  // blocks per product
    unsigned long long* ticket;
    uint64_t ticket_base, epoch;
    uint32_t* err;
};

constexpr uint32_t kWideCarryChunks = 256;  // 256-bit chunks per carry block
// Carry blocks of a product with out_cap output elements.
__host__ __device__ inline uint32_t wide_carry_blocks(size_t out_cap, int out_fmt) {
    const uint64_t limbs = out_fmt == kFmtLimb64 ? out_cap : ((uint64_t)out_cap * 28 + 63) / 64;
    return (uint32_t)((limbs + 4 * kWideCarryChunks - 1) / (4 * kWideCarryChunks));
}

// Split of 2^log_n 64-bit digits: the tuned one of 2^(log_n + 1) 32-bit digits
// (bgpu_set_split, bgpu_set_batch_split) where its kernels are built, else the
// built-in one.  log_n2 == 0: no five-prime transform of this length.
TransformShape wide_shape(int log_n, bool batch);
cudaError_t upload_wide_consts(int set, const NttConsts& c);
extern const char* const kWideKernelNames[kNttLaunches];

// The four launches of `count` products of 2^log_n points (64-bit digits of
// both operands together at most 2^log_n + 1); each product's carry scan has
// `bpp` blocks (tickets).
cudaError_t launch_wide_product(const NttConsts& host, const ProductDesc* descs, const ProductDesc& one,
                                uint32_t count, bool square, int log_n, int out_fmt, uint32_t bpp,
                                const CarryLaunch& cl, cudaStream_t st, cudaEvent_t* ev);

// The same for any number of products in the device array `descs`, in pieces
// that fit a launch grid, all on one ticket sequence from cl.ticket_base.
cudaError_t launch_wide_batch(const NttConsts& host, const ProductDesc* descs, uint32_t count, bool square, int log_n,
                              int out_fmt, uint32_t bpp, const CarryLaunch& cl, cudaStream_t st);

}  // namespace bgpu
