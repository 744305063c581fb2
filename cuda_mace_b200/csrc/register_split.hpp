// Register splits between the halves of a block (setmaxnreg); host arithmetic.
#pragma once

namespace cmace {

// Whether a block launched with regs registers a thread holds a split into two halves of its threads.  setmaxnreg.inc takes
// from what the block was launched with, not from the SM's registers, and waits without a limit for the rest.
constexpr bool register_split_fits(int regs, int threads, int first_half, int second_half) {
  return (first_half + second_half) * (threads / 2) <= regs * threads;
}

}  // namespace cmace
