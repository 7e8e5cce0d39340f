// Index arithmetic of the GEMM kernels that the CPU unit tests (tests/cpp/runtime_unit.cpp) check as well. No CUDA types.
#pragma once

namespace rocshmem {
namespace kernels {

// First row of the second 128-row box of B of a 256-column tile with `cols` valid columns whose first box starts at row
// `first`. A width that is an odd multiple of 128 ends in a tile whose second half does not exist: it then names its
// first box twice, because the block scales of rows behind it may lie past their array (its sums are not stored).
// (To choose the scales' row in the accumulate warps instead cost 4 - 5 % at 512 x 4096 x 4096 to 2048 x 7168 x 2048.)
constexpr int second_box(int first, int cols) { return cols > 128 ? first + 128 : first; }

// Fewest CTAs that may share the K of a 128 x 128 tile of a bf16 product (gemm_split_core.cuh). One, i.e. twice as many
// SMs reading the weight as the one-CTA kernel has, pays for one block of rows: weights from memory, 75 to 144 tiles, 1 to
// 128 rows, K 1024 / 2048 / 4096 take 0.88 - 1.06 / 0.84 - 0.97 / 0.74 - 0.95 of its time, K 512 up to 1.19. With more rows
// the two-CTA kernel moves half the operand bytes on the same SMs: one CTA a tile took 1.00 - 1.04 of its time (96 to
// 144 tiles, K 1024 to 8192; with the operands in L2 1.00 - 1.06).
constexpr int split_least_bf16(int m, int k) { return m <= 128 && k >= 1024 ? 1 : 2; }

// Whether a block whose warps hand registers to one another (setmaxnreg) may be launched: `compiled` is what the kernel
// really uses per thread, `launch` what the hand-over was laid out for and gives back at the end. With fewer registers
// the instruction that takes more would wait for ever.
constexpr bool hand_over_fits(int compiled, int launch, int giving_warps, int giving, int taking_warps, int taking) {
  return compiled == launch && giving_warps * giving + taking_warps * taking <= (giving_warps + taking_warps) * compiled;
}

}  // namespace kernels
}  // namespace rocshmem
