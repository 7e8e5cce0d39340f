// Index arithmetic of the GEMM kernels that the CPU unit tests (tests/cpp/runtime_unit.cpp) check as well. No CUDA types.
#pragma once

namespace rocshmem {
namespace kernels {

// The 128-row box of B whose block scales a thread reads that adds up half `half` of a 256-column tile (128 columns a half)
// with `cols` valid columns. A product whose width is an odd multiple of 128 ends in a tile whose second half does
// not exist: its sums are not stored, and the scale row behind it may lie past the array.
constexpr int b_scale_box(int half, int cols) { return half * 128 < cols ? half : 0; }

// Whether a block whose warps hand registers to one another (setmaxnreg) may be launched: `compiled` is what the kernel
// really uses per thread, `launch` what the hand-over was laid out for and gives back at the end. With fewer registers
// the instruction that takes more would wait for ever.
constexpr bool hand_over_fits(int compiled, int launch, int giving_warps, int giving, int taking_warps, int taking) {
  return compiled == launch && giving_warps * giving + taking_warps * taking <= (giving_warps + taking_warps) * compiled;
}

}  // namespace kernels
}  // namespace rocshmem
