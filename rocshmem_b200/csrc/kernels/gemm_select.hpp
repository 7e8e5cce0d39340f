// Index arithmetic of the GEMM kernels that the CPU unit tests (tests/cpp/runtime_unit.cpp) check as well. No CUDA types.
#pragma once

namespace rocshmem {
namespace kernels {

// The 128-row box of B whose block scales a thread reads that adds up half `half` of a 256-column tile (128 columns a half)
// with `cols` valid columns. A product whose width is an odd multiple of 128 ends in a tile whose second half does
// not exist: its sums are not stored, and the scale row behind it may lie past the array.
constexpr int b_scale_box(int half, int cols) { return half * 128 < cols ? half : 0; }

}  // namespace kernels
}  // namespace rocshmem
