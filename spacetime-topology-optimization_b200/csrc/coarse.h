// The coarsest level's direct solve: block elimination of the grid's lines in odd-even
// order (coarse.cu).
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"
#include "hier.h"

namespace stt {

// Plans the factor for the coarsest level (co.n, co.tree, co.B, co.nb, co.by_col).
void coarse_plan(const LevelDesc& c, int d, int hrows, CoarseDesc& co);
// Assembles the coarse matrix from the level's FP64 stencil and factorises it on `st`.
int coarse_factor(const stt_hier* h, cudaStream_t st);
// x = A^{-1} b (T = float or double; FP64 arithmetic) for nrows batch rows; only for co.tree.
template <typename T>
int coarse_tree_solve(const stt_hier* h, int nrows, const T* b, T* x, long long rs, const RowState* rst,
                      cudaStream_t st);

}  // namespace stt
