// Device functions shared by the stand-alone kernels and the fused decode step, so that
// both execute literally the same arithmetic.
#pragma once
#include "lt_common.cuh"

namespace lt {

// NeoX half-split rotation of one (x1, x2) pair of a head at integer position `pos`:
// freq = powf(theta, -(2j)/hd), ang = pos * freq, o1 = x1*cos - x2*sin, o2 = x1*sin + x2*cos.
// The reference kernel's source leaves the two output expressions to nvcc's default
// contraction; compiled for sm_100a it comes out as
//     o1 = fma(x1, cos, -(x2*sin))      o2 = fma(x2, cos, x1*sin)
// (found by comparing the explicit candidates with the reference's own kernel bit for bit on
// the GPU, which the parity tests keep doing).  It is written out here so that no context can
// change it.  The angle part depends only on (j, pos), so a fused kernel may evaluate it before
// its input has arrived.
__device__ __forceinline__ void rope_trig(int j, int hd, float theta, int pos, float& c, float& s) {
    float p = (float)pos;
    float freq = powf(theta, -(2.0f * (float)j) / (float)hd);
    float ang = p * freq;
    c = cosf(ang);
    s = sinf(ang);
}
__device__ __forceinline__ void rope_rotate(float x1, float x2, float c, float s, float& o1, float& o2) {
    o1 = __fmaf_rn(x1, c, -__fmul_rn(x2, s));
    o2 = __fmaf_rn(x2, c, __fmul_rn(x1, s));
}
__device__ __forceinline__ void rope_pair(float x1, float x2, int j, int hd, float theta, int pos, float& o1,
                                          float& o2) {
    float c, s;
    rope_trig(j, hd, theta, pos, c, s);
    rope_rotate(x1, x2, c, s, o1, o2);
}

// ---- RMSNorm and quantiser over a vector in shared memory, for kernels that fuse them as a prologue
// sum of squares in the declared 256-lane order; blocks of at least 256 threads
__device__ __forceinline__ float block_rms_sumsq(const float* sF, int N, float* sred) {
    const int t = threadIdx.x;
    float local = 0.0f;
    if (t < 256) {
        int j = t;
#pragma unroll 1
        for (; j + 768 < N; j += 1024) {    // four reads on their way per step of the chain
            const float a = sF[j], b = sF[j + 256], c = sF[j + 512], d = sF[j + 768];
            local = __fmaf_rn(a, a, local);
            local = __fmaf_rn(b, b, local);
            local = __fmaf_rn(c, c, local);
            local = __fmaf_rn(d, d, local);
        }
        for (; j < N; j += 256) local = __fmaf_rn(sF[j], sF[j], local);
    }
    if (t < 256) sred[t] = local;
    __syncthreads();
    if (t < 32) {
        const float* p = sred;   // levels 128, 64, 32 in the declared pairing, then 16 .. 1
        const float a = __fadd_rn(__fadd_rn(p[t], p[t + 128]), __fadd_rn(p[t + 64], p[t + 192]));
        const float b = __fadd_rn(__fadd_rn(p[t + 32], p[t + 160]), __fadd_rn(p[t + 96], p[t + 224]));
        const float v = warp_tree_sum(__fadd_rn(a, b));
        if (t == 0) sred[256] = v;
    }
    __syncthreads();
    return sred[256];
}

// quantise N floats of shared memory (optionally (x*inv)*w first) into sXq / sXd; all warps.  Eight threads per block, four values
// each (16-byte aligned vectors).  A lane per value with divisions took three times the instructions, which the CTAs of an SM
// share: a GEMV of 6144 x 4096 behind a norm 12.7 us, now 10.3 (7.2 without the norm).
__device__ __forceinline__ void block_quant(const float* sF, const float* sW, float inv, int N, int8_t* sXq,
                                            __half* sXd) {
    const int nquad = N >> 2;      // a multiple of 8: the eight threads of a block are in or out together
    for (int i0 = threadIdx.x & ~31; i0 < nquad; i0 += blockDim.x) {
        const int i = i0 + (threadIdx.x & 31);
        float4 x = i < nquad ? ((const float4*)sF)[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (sW != nullptr && i < nquad) {
            const float4 w = ((const float4*)sW)[i];
            x.x = __fmul_rn(__fmul_rn(x.x, inv), w.x); x.y = __fmul_rn(__fmul_rn(x.y, inv), w.y);
            x.z = __fmul_rn(__fmul_rn(x.z, inv), w.z); x.w = __fmul_rn(__fmul_rn(x.w, inv), w.w);
        }
        unsigned m = max(max(__float_as_uint(fabsf(x.x)), __float_as_uint(fabsf(x.y))),
                         max(__float_as_uint(fabsf(x.z)), __float_as_uint(fabsf(x.w))));
#pragma unroll
        for (int s = 4; s > 0; s >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, s));
        const __half dh = q8_scale(__uint_as_float(m));
        const float dq = __half2float(dh), r = q8_reciprocal(dq);
        const int q0 = q8_value(x.x, dq, r), q1 = q8_value(x.y, dq, r), q2 = q8_value(x.z, dq, r), q3 = q8_value(x.w, dq, r);
        if (i < nquad) {
            ((char4*)sXq)[i] = make_char4((signed char)q0, (signed char)q1, (signed char)q2, (signed char)q3);
            if ((i & 7) == 0) sXd[i >> 3] = dh;
        }
    }
}

}  // namespace lt
