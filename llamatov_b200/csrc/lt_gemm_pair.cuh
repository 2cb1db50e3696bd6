// The Q8_0 GEMM with 32-column tiles and scale products on the tensor cores (lt_gemm_pair.cu), as lt_q8_gemm_tc reaches it.
#pragma once
#include <cuda.h>

#include "lt_common.cuh"

namespace lt {
namespace tc {

// 2-D byte tensor [rows][K] (row-major), box = box_k bytes x box_rows rows, hardware swizzle of box_k bytes
int make_map(CUtensorMap* m, const void* ptr, int rows, int K, int box_k, int box_rows);

namespace pair {
struct Args {
    const int8_t *Wq, *Xq;
    const uint16_t *Wd, *Xd;
    const float* Resid;
    int resid_ld;
    float* Y;
    int M, K, T;
};
bool fits(int M, int K, int T);
double cost(int M, int K, int T, int sms);   // microseconds, as measured
int run(const Args& a, cudaStream_t s);      // K a multiple of 128
}  // namespace pair
}  // namespace tc
}  // namespace lt
