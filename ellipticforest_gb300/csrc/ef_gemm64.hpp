// Merges of the build with FP64-accurate tensor-core products (ef_gemm64.cu).
#pragma once

#include <cuda_runtime.h>

#include <climits>
#include <cstddef>

#include "ef_kernels.cuh"

namespace efgb {

// one device pointer per batch item, `stride` bytes apart
struct PtrTable {
    const void* p;
    long long stride;
};

// A matrix per batch item: entry (r, k) at base[b] + off + r ld + k, rows from rs on shifted by dr and columns
// from ks on by dk (blocks that are not adjacent in memory)
struct MatView {
    PtrTable base;
    long long off;
    int ld;
    int rs = INT_MAX, ks = INT_MAX;
    long long dr = 0, dk = 0;
};

// Merges of `cnt` nodes of child side s whose X, H and T_LHS are gathered: S and X^{-1} into RHS, T += H S.
// info[i] != 0 where the elimination met a bad pivot or its residual is not that of a pivoted one: the
// caller then merges with the pivoted LU.  ws: merge64_workspace bytes; err: set when a wait gave up.
bool merge64_supported(int s);
size_t merge64_workspace(int cnt, int s);
void merge64(cudaStream_t st, const MergeItem* items, int cnt, int s, int* info, char* ws, int* err);

// A <- A^-1 of one h x h row-major matrix in place (A: device address holding its pointer) by the same block
// elimination; info as above except for the residual, which is the caller's to check.  tmp: invert64_tmp doubles.
size_t invert64_workspace(int h);
size_t invert64_tmp(int h);
void invert64(cudaStream_t st, double* const* A, double* const* tmp, int h, int* info, char* ws, int* err);

}  // namespace efgb
