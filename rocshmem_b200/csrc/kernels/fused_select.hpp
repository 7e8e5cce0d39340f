// What the fused tensor-parallel calls do with operands that share memory. Pure host logic, no CUDA types: the launchers
// in fused_kernels.cu and the CPU unit tests (tests/cpp/runtime_unit.cpp) share it.
#pragma once

#include <cstddef>
#include <cstdint>

namespace rocshmem {
namespace kernels {

// A piece of device memory; one without bytes overlaps nothing.
struct Span {
  const void *ptr;
  size_t bytes;
};

inline bool overlaps(const Span &a, const Span &b) {
  const uintptr_t x = reinterpret_cast<uintptr_t>(a.ptr), y = reinterpret_cast<uintptr_t>(b.ptr);
  return a.bytes != 0 && b.bytes != 0 && x < y + b.bytes && y < x + a.bytes;
}

// all-gather -> GEMM on a team of one. The rows become the input buffer's content (`keep`) first, then the result is
// written. The kernel reads the rows where they are and writes `keep` and the result side by side, which is the same
// only as long as none of the three shares memory with another and `keep` shares none with the weight.
struct AlonePlan {
  bool rows_aside;   // rows -> gather buffer before the kernel, which reads them there
  bool keep_first;   // rows (from where the kernel reads them) -> keep before the kernel, which then copies nothing
};

inline AlonePlan plan_alone(const Span &rows, const Span &keep, const Span &weight, const Span &result) {
  return AlonePlan{overlaps(rows, result) || overlaps(rows, keep), overlaps(keep, result) || overlaps(keep, rows) || overlaps(keep, weight)};
}

}  // namespace kernels
}  // namespace rocshmem
