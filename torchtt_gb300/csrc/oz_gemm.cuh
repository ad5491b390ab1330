// Large FP64 contractions on the tcgen05 tensor cores: the digit products of contract_emu.cuh with the
// digits made once per operand element, in a launch of their own, and multiplied by tcgen05.mma from
// shared memory that bulk copies fill (see oz_gemm.cu).
#pragma once

#include "contract.cuh"

namespace ttgb {

// Whether oz_contract takes the contraction.
bool oz_takes(const ContractDesc& d);

// Upper bound of the workspace of an oz_contract that oz_takes, in bytes: elements is the number of elements of
// its larger operand (of all batch entries that differ).
double oz_workspace_bound(double elements);

// K units of its split (a split's range is a multiple of this).
constexpr int kOzChunk = 128;

// Output tiles of a launch (for the split-K choice).
int64_t oz_tiles(const ContractDesc& d);

// C (+)= alpha A B as launch_tiles' other kernels: splitk ranges of kchunk are added atomically into C
// (which already holds beta C), one range writes alpha A B + beta C.
// False, with nothing launched, when there is no memory for the digits.
bool oz_contract(const ContractDesc& d, int splitk, int kchunk, cudaStream_t s);

// The calling host thread's error word (pinned): a kernel launched by it sets the word when one of its bounded
// waits gave up.
int* wait_error_word();
// Whether the word was set, which it then no longer is. Covers the kernels that have completed.
bool take_wait_error();

}  // namespace ttgb
