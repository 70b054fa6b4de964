// Which elements a tensor's magnitude is sampled from (tc_gemm.cu); plain C++, so that it can be checked without a GPU.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define MCL_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define MCL_HOST_DEVICE inline
#endif

namespace mcl {

constexpr int kSampleUnits = 4096;          // units of 4 consecutive elements

// Unit number that sample u stands for: one unit out of each run of `step`, at the offset frac(u / golden ratio) of the run.  At a fixed
// offset a step that is a multiple of the row length (8192 x 288, 4096 x 32000) would see the same four columns of every row.
MCL_HOST_DEVICE long long sample_unit(long long u, long long step) {
    const uint32_t turn = (uint32_t)u * 0x9E3779B1u;
    return u * step + (long long)(((uint64_t)turn * (uint64_t)step) >> 32);
}

}  // namespace mcl
