// Launches of the two-CTA linear kernel (gemm_pair.cu).
#pragma once
#include "common.cuh"
#include "gemm_common.cuh"

// Pairs of CTAs the device runs at once.
int linear_pair_capacity();
// p.grid: two CTAs per pair; a.n_tiles counts tiles of 256 weight rows.
void launch_linear_pair(const LinearPlan& p, const gemm::LinearArgs& a, cudaStream_t s);
