// Few-row products on CUDA warps' matrix instructions; see gemm_rows.cu.
#pragma once
#include "epilogue.cuh"

// The kernel takes a step's product of M rows: one plain product or one with column groups, in a 16-bit format.
bool arcb_gemm_rows_applies(const void* a16, const void* w16, const GemmEpilogue& ep, int K, int act_f16);
int arcb_launch_gemm_rows(const void* a16, const void* w16, const GemmEpilogue& ep, int K, int act_f16, cudaStream_t stream);
