// mul_direct.cuh -- direct (schoolbook) products of short operands.
#pragma once
#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

#include "ntt_kernels.cuh"

namespace precgpu {

// batch form: one product per group of 32 or more threads, longer operand
// up to kDirectBatchMax limbs; classes 0 .. kDirectClasses-1 by that length
constexpr int kDirectClasses = 4;
constexpr uint64_t kDirectBatchMax = 512;

// single product over the whole GPU: longer operand up to kDirectGridMax limbs
constexpr uint64_t kDirectGridMax = 4096;

// class of a batch product, or -1: the transform is faster (see the rule)
int direct_class(uint64_t la, uint64_t lb);
// whether a single device product runs directly
bool direct_single(uint64_t la, uint64_t lb);
// scratch bytes of a single direct product (column sums)
size_t direct_scratch_bytes(uint64_t la, uint64_t lb);

void launch_direct_batch(const SmallDesc* d_descs, int count, int cls, cudaStream_t st);
// counter: one device word, zero before the first call, left zero by every
// call; calls that share it must not overlap
void launch_direct_single(const uint64_t* a, uint64_t la, const uint64_t* b, uint64_t lb, uint64_t* out,
                          uint8_t* scratch, uint32_t* counter, cudaStream_t st);
int configure_direct();

}  // namespace precgpu
