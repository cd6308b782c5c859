// Resident step kernel of the batched engine: one cooperative launch advances
// every instance by many steps (until the shared list rebuild or the step
// target), with grid barriers in the place of the kernel boundaries.
#pragma once

#include "hm2d_run.cuh"

namespace tdem {
namespace hm {

// Threads of the one block per SM: FP32 takes 128 registers, FP64 255 (its
// pipe, not the number of warps, bounds it).
template <class T>
constexpr int kBatchRunBlock = sizeof(T) == 4 ? 512 : 256;

// Stage of one tile in a thread's shared memory: the pipelined force pass
// (three heads, two own states, two sets of three partners, two remainders,
// two sets of bond words) and the strain pass share it.
inline size_t batch_run_smem(int bmax, bool prem, bool fp32) {
  if (!fp32) return 0;
  constexpr int block = kBatchRunBlock<float>;
  const size_t force = async_smem(block, prem) + (bmax > 0 ? async_bond_smem(block, bmax) : 0);
  const size_t strain = bmax > 0 ? strain_smem_bytes(block) : 0;
  return force > strain ? force : strain;
}

template <class T>
using BatchRunFn = void (*)(Bufs<T>, cudaGraphConditionalHandle, cudaGraphConditionalHandle, int, int, int, int, int,
                            long long);
template <class T>
BatchRunFn<T> batch_run_fn();

}  // namespace hm
}  // namespace tdem
