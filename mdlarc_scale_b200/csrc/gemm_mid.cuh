// Products of a few dozen to 256 rows on tcgen05 tiles of the transposed product; see gemm_mid.cu.
#pragma once
#include "epilogue.cuh"

bool arcb_gemm_mid_applies(const void* a16, const void* w16, const GemmEpilogue& ep, int K, int act_f16);
int arcb_launch_gemm_mid(const void* a16, const void* w16, const GemmEpilogue& ep, int K, int act_f16, cudaStream_t stream);
