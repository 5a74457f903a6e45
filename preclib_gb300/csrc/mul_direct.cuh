// mul_direct.cuh -- direct (schoolbook) products of short operands.
#pragma once
#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

#include "ntt_kernels.cuh"

namespace precgpu {

// batch form: one product per group of 32 or more threads, longer operand
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
// empty).  Direct where it measured below the single-CTA transform (ns per
// product of a large batch, direct / transform, equal operands of n limbs):
// 16: 1.2 / 18.7, 32: 1.8 / 18.8, 64: 3.2 / 21.0, 96: 6.2 / 23.5 (8.9 in the
// class up to 128 limbs), 128: 11.4 / 24.6, 192: 29.1 / 27.8, 256: 37.1 / 29.0, 512: 139 / 70.  The direct time
// goes with the shorter operand, the transform's with the sum: operands up to
// 256 limbs cross near 180 x 180 limbs, operands up to 512 limbs at a
// shorter one of about 100 limbs (27 ns against 29 of the 2^10-point
// transform).
__host__ __device__ inline int direct_class(uint64_t la, uint64_t lb) {
    const uint64_t hi = la > lb ? la : lb, lo = la > lb ? lb : la;
    if (lo == 0) return -1;
    if (hi <= 96) return hi <= 64 ? 0 : 1;
    if (hi <= 128) return 2;
    if (hi <= 256) return lo <= 160 ? 3 : -1;
    return hi <= kDirectBatchMax && lo <= 96 ? 4 : -1;
}
// whether a single device product runs directly
bool direct_single(uint64_t la, uint64_t lb);
// scratch bytes of a single direct product (column sums)
size_t direct_scratch_bytes(uint64_t la, uint64_t lb);

// Every item's index into its class's list: lists[cls * count ..], their
// lengths in n[kDirectClasses], zero before.
void launch_direct_lists(const DirectItem* d_items, int count, uint32_t* lists, uint32_t* n, cudaStream_t st);
// Products of class `cls`: `count` items, or the *n items (at most `count`)
// whose indices `list` holds.
void launch_direct_batch(const DirectItem* d_items, int count, int cls, cudaStream_t st,
                         const uint32_t* list = nullptr, const uint32_t* n = nullptr);
// counter: one device word, zero before the first call, left zero by every
// call; calls that share it must not overlap
void launch_direct_single(const uint64_t* a, uint64_t la, const uint64_t* b, uint64_t lb, uint64_t* out,
                          uint8_t* scratch, uint32_t* counter, cudaStream_t st);
int configure_direct();

}  // namespace precgpu
