// 32-bit products on the bf16 matrix instructions; see gemm_split.cu.
#pragma once
#include "epilogue.cuh"

bool arcb_gemm_split_applies(const void* a, const void* w, const GemmEpilogue& ep, int K);
int arcb_launch_gemm_split(const void* a, const void* w, const GemmEpilogue& ep, int K, cudaStream_t stream);
