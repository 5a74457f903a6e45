// mul_direct.cuh -- direct (schoolbook) products of short operands.
#pragma once
#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

#include "ntt_kernels.cuh"

namespace precgpu {

// batch form: one product per group of 16 to 128 threads, longer operand
// up to kDirectBatchMax limbs; classes 0 .. kDirectClasses-1 by that length
constexpr int kDirectClasses = 5;
constexpr uint64_t kDirectBatchMax = 512;

// single product over the whole GPU: longer operand up to kDirectGridMax limbs
constexpr uint64_t kDirectGridMax = 4096;

// One product of a batch: the layout of prec_gpu_product_t, so that a batch of
// direct products alone takes the caller's array as it is.
struct DirectItem {
    const uint64_t* a;
    uint64_t la;
    const uint64_t* b;
    uint64_t lb;
    uint64_t* out;
};

// Class of a batch product, or -1: the transform is faster (or an operand is
// empty).  Direct where it measured below the single-CTA transform.  The
// direct time goes with the class and the shorter operand, the transform's
// with the points (ns per product of a large batch; 13.1 for 2^9 points, a sum of
// up to 256 limbs, 19.9 for 2^10, 37.8 for 2^11):
//   up to 128 limbs: 16 x 16 1.2, 32 1.8, 64 3.2, 96 6.2, 128 11.4
//   up to 256, shorter operand 32: 7.7, 64: 13.3, 96: 18.6, 112: 21.3, 160: 28.9
//   up to 512, shorter operand 32: 11.5 - 13.8, 48: 15.4 - 18.5, 64: 19.0 -
//   23.3, 80: 28.2, 96: 33.3
__host__ __device__ inline int direct_class(uint64_t la, uint64_t lb) {
    const uint64_t hi = la > lb ? la : lb, lo = la > lb ? lb : la;
    if (lo == 0) return -1;
    if (hi <= 96) return hi <= 64 ? 0 : 1;
    if (hi <= 128) return 2;
    if (hi <= 256) return lo <= (hi + lo <= 256 ? 64 : 104) ? 3 : -1;
    return hi <= kDirectBatchMax && lo <= (hi + lo <= 512 ? 52 : 96) ? 4 : -1;
}
// whether a single device product runs directly
bool direct_single(uint64_t la, uint64_t lb);
// scratch bytes of a single direct product (column sums)
size_t direct_scratch_bytes(uint64_t la, uint64_t lb);

// CTAs that take `count` items `per` at a time, at most `cap`.  A CTA's items are
// per * block, and per * (CTAs) further each round: 64-bit, as a batch may hold
// 2^31 - 1 products and the round past the last one lies beyond that.
__host__ __device__ inline int direct_ctas(int count, int per, int cap) {
    const int64_t n = ((int64_t)count + per - 1) / per;
    return n < cap ? (int)n : cap;
}
__host__ __device__ inline int64_t direct_first(uint32_t block, int per) { return (int64_t)block * per; }

// Every item's index into its class's list: lists[cls * count ..], their
// lengths in n[kDirectClasses], zero before.
void launch_direct_lists(const DirectItem* d_items, int count, uint32_t* lists, uint32_t* n, cudaStream_t st);
// Products of class `cls`: `count` items, or the *n items (at most `count`)
// whose indices `list` holds.
void launch_direct_batch(const DirectItem* d_items, int count, int cls, cudaStream_t st,
                         const uint32_t* list = nullptr, const uint32_t* n = nullptr);
// counter: one device word, zero before the first call, left zero by every
// call; calls that share it must not overlap.  A carry out of the product sets
// kDevErrCarry in *err.
void launch_direct_single(const uint64_t* a, uint64_t la, const uint64_t* b, uint64_t lb, uint64_t* out,
                          uint8_t* scratch, uint32_t* counter, int* err, cudaStream_t st);
int configure_direct();

}  // namespace precgpu
