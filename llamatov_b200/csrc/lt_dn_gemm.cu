// Linear over a block of token rows, Y[t][n] = epilogue(sum_k W[n][k] X[t][k]).
//
// bf16 (k_gemm_tc): tcgen05.mma kind::f16, fp32 accumulators in tensor memory.  A tile is MA x 128 weight rows (the
// MMA's M: tensor-memory lanes) by NT tokens (its N: columns); with MA = 2 the second 128 rows are the "up" rows that
// belong to the first 128 "gate" rows, so that act(gate) * up is formed where both accumulators are.  An epilogue
// thread owns one weight row: bias, activation and layer scale are per-thread constants, and the 32 lanes of a
// warp store 32 consecutive outputs of a token.
//   warp 8 : producer, TMA tiles of 64 k (128-byte rows, hardware swizzle) into a ring of shared-memory stages
//   warp 9 : one thread issues the MMAs; two accumulator sets, so the next tile's MMAs run under this tile's epilogue
//   warps 0-7 : epilogue
// fp32 (k_gemm_f32): register-blocked tiles on the CUDA cores, every product and sum an fp32 fused multiply-add.
#include "lt_dn_common.cuh"
#include "lt_tc.cuh"

namespace lt {
namespace dn {

using namespace tc;

struct GemmP {
    void* Y;
    int* status;
    int M, K, T, ldy;
    int row_tiles, t_tiles;
    int up_row;          // first "up" row (MA = 2)
    lt_dn_epilogue epi;
};

constexpr int BK = 64;   // k elements of a stage (128 bytes)

template <int NT, int MA>
struct GemmCfg {
    static constexpr int W_STAGE = MA * 128 * 128;
    static constexpr int X_STAGE = NT * 128;
    static constexpr int STAGE = W_STAGE + X_STAGE;
    static constexpr int NSTAGE = (200 * 1024) / STAGE > 8 ? 8 : (200 * 1024) / STAGE;
    static constexpr int ACC_COLS = MA * NT;
    static constexpr int TMEM = 2 * ACC_COLS < 32 ? 32 : 2 * ACC_COLS;
    static constexpr int EW = 8;
    static constexpr int THREADS = (EW + 2) * 32;
    static constexpr int SMEM = 1024 + NSTAGE * STAGE + 1024;
    static_assert(TMEM <= 512 && (TMEM & (TMEM - 1)) == 0, "tensor memory columns");
    static_assert(X_STAGE % 1024 == 0, "stages keep 1024-byte alignment");
};

struct GemmBars {
    unsigned long long full[8], empty[8], tfull[2], tempty[2];
    unsigned tmem_base;
    int abort_flag;
};

// D[tmem] (+)= A[smem] * B[smem], bf16 x bf16 -> fp32
__device__ __forceinline__ void mma_bf16(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, bool acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"((int)acc)
        : "memory");
}

template <int NT, int MA>
__global__ void __launch_bounds__(GemmCfg<NT, MA>::THREADS, 1)
k_gemm_tc(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const __grid_constant__ GemmP P) {
    using C = GemmCfg<NT, MA>;
    constexpr int NS = C::NSTAGE;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    GemmBars* B = (GemmBars*)(base + NS * C::STAGE);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles = P.row_tiles * P.t_tiles;
    const int nk = (P.K + BK - 1) / BK;
    volatile int* abort_flag = &B->abort_flag;

    if (tid == 0) {
        for (int s = 0; s < NS; s++) {
            mbar_init(&B->full[s], 1);
            mbar_init(&B->empty[s], 1);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(&B->tfull[s], 1);
            mbar_init(&B->tempty[s], C::EW);
        }
        B->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == C::EW + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&B->tmem_base)),
                     "r"((unsigned)C::TMEM)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = B->tmem_base;

    if (warp == C::EW) {
        if (lane == 0) {
            unsigned it = 0;
            for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
                const int rt = tile % P.row_tiles, tt = tile / P.row_tiles;
                for (int kb = 0; kb < nk; kb++, it++) {
                    const int s = it % NS;
                    unsigned char* st = base + s * C::STAGE;
                    mbar_wait<32>(&B->empty[s], ((it / NS) & 1) ^ 1, abort_flag, P.status);
                    mbar_expect_tx(&B->full[s], C::STAGE);
                    tma_load_2d(st, &tmW, kb * BK, rt * 128, &B->full[s]);
                    if (MA == 2) tma_load_2d(st + 128 * 128, &tmW, kb * BK, P.up_row + rt * 128, &B->full[s]);
                    tma_load_2d(st + C::W_STAGE, &tmX, kb * BK, tt * NT, &B->full[s]);
                }
            }
        }
    } else if (warp == C::EW + 1) {
        if (lane == 0) {
            // D fp32, A and B bf16, both K-major, N = NT, M = 128
            constexpr unsigned idesc =
                (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(NT >> 3) << 17) | ((unsigned)(128 >> 4) << 24);
            const unsigned long long w0 = smem_desc<4>(smem_u32(base));
            const unsigned long long x0 = smem_desc<4>(smem_u32(base) + C::W_STAGE);
            unsigned it = 0, n = 0;
            for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, n++) {
                const unsigned slot = n & 1;
                mbar_wait<32>(&B->tempty[slot], ((n >> 1) & 1) ^ 1, abort_flag, P.status);
                tc_fence_after();
                const unsigned d = tmem + slot * C::ACC_COLS;
                for (int kb = 0; kb < nk; kb++, it++) {
                    const unsigned s = it % NS;
                    mbar_wait<0>(&B->full[s], (it / NS) & 1, abort_flag, P.status);
                    tc_fence_after();
                    const unsigned long long wd = w0 + (unsigned long long)(s * (C::STAGE >> 4));
                    const unsigned long long xd = x0 + (unsigned long long)(s * (C::STAGE >> 4));
#pragma unroll
                    for (int j = 0; j < BK / 16; j++) {
#pragma unroll
                        for (int a = 0; a < MA; a++)
                            mma_bf16(d + a * NT, wd + a * (128 * 128 >> 4) + 2 * j, xd + 2 * j, idesc, kb > 0 || j > 0);
                    }
                    mma_commit(&B->empty[s]);
                }
                mma_commit(&B->tfull[slot]);
            }
        }
    } else {
        const int q = warp & 3, cg = warp >> 2;
        constexpr int CW = NT / 2;                // columns of this warp
        unsigned n = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, n++) {
            const int rt = tile % P.row_tiles, tt = tile / P.row_tiles;
            const int row = rt * 128 + q * 32 + lane;
            const bool row_ok = row < P.M;
            const int t0 = tt * NT + cg * CW;
            const unsigned slot = n & 1;
            const RowEpi re = row_epi(P.epi, row_ok ? row : 0);
            mbar_wait<32>(&B->tfull[slot], (n >> 1) & 1, abort_flag, P.status);
            tc_fence_after();
            const unsigned ta = tmem + ((unsigned)(q * 32) << 16) + slot * C::ACC_COLS + cg * CW;
#pragma unroll 1
            for (int c0 = 0; c0 < CW; c0 += 16) {
                if (t0 + c0 >= P.T) break;        // the same for the whole warp
                int v[MA][16];
#pragma unroll
                for (int a = 0; a < MA; a++) tmem_ld<16>(ta + a * NT + c0, v[a]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int a = 0; a < MA; a++)
#pragma unroll
                    for (int c = 0; c < 16; c += 4) reg_fence4(&v[a][c]);
                if (row_ok) {
                    if (MA == 2) {
                        float f[16];
                        if (P.epi.out_f32) {
#pragma unroll
                            for (int c = 0; c < 16; c++)
                                f[c] = glu_f(P.epi, __int_as_float(v[0][c]), __int_as_float(v[MA - 1][c]));
                            float* y = (float*)P.Y + (long)(t0 + c0) * P.ldy + row;
#pragma unroll
                            for (int c = 0; c < 16; c++)
                                if (t0 + c0 + c < P.T) y[(long)c * P.ldy] = f[c];
                        } else {
                            glu_bf16(P.epi, v[0], v[MA - 1], f);
                            bf16* y = (bf16*)P.Y + (long)(t0 + c0) * P.ldy + row;
#pragma unroll
                            for (int c = 0; c < 16; c++)
                                if (t0 + c0 + c < P.T) y[(long)c * P.ldy] = from_f<bf16>(f[c]);
                        }
                    } else if (P.epi.kind == LT_DN_RESID) {
                        float* y = (float*)P.Y + (long)(t0 + c0) * P.ldy + row;
                        float old[16];
#pragma unroll
                        for (int c = 0; c < 16; c++)
                            if (t0 + c0 + c < P.T) old[c] = y[(long)c * P.ldy];
#pragma unroll
                        for (int c = 0; c < 16; c++)
                            if (t0 + c0 + c < P.T)
                                y[(long)c * P.ldy] = fmaf(re.ls, __int_as_float(v[0][c]) + re.bias, old[c]);
                    } else {
                        float f[16];
#pragma unroll
                        for (int c = 0; c < 16; c++) f[c] = __int_as_float(v[0][c]);
                        if (P.epi.tail != nullptr && row >= P.epi.tail_from) {
                            epi_values<false>(re, f);
                            float* y = P.epi.tail + (long)(t0 + c0) * P.epi.ldtail + row - P.epi.tail_from;
#pragma unroll
                            for (int c = 0; c < 16; c++)
                                if (t0 + c0 + c < P.T) y[(long)c * P.epi.ldtail] = f[c];
                        } else if (P.epi.out_f32) {
                            epi_values<false>(re, f);
                            float* y = (float*)P.Y + (long)(t0 + c0) * P.ldy + row;
#pragma unroll
                            for (int c = 0; c < 16; c++)
                                if (t0 + c0 + c < P.T) y[(long)c * P.ldy] = f[c];
                        } else {
                            epi_values<true>(re, f);
                            bf16* y = (bf16*)P.Y + (long)(t0 + c0) * P.ldy + row;
#pragma unroll
                            for (int c = 0; c < 16; c++)
                                if (t0 + c0 + c < P.T) y[(long)c * P.ldy] = from_f<bf16>(f[c]);
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&B->tempty[slot]);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag && tid == 0) {     // a wait ran out: let copies in flight land before the CTA leaves
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) {
        }
    }
    __syncthreads();
    if (warp == C::EW + 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((unsigned)C::TMEM) : "memory");
    }
}

// [rows][K] bf16 with row stride ld, box 64 k x box_rows
static int make_map_bf16(CUtensorMap* m, const void* ptr, long rows, int K, int ld, int box_rows) {
    encode_fn_t fn = encode_fn();
    if (fn == nullptr) {
        set_error("lt_dn_linear: cuTensorMapEncodeTiled is not available from this driver");
        return LT_ERR_CUDA;
    }
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("lt_dn_linear: cuTensorMapEncodeTiled failed (%d) for rows=%ld K=%d ld=%d", (int)r, rows, K, ld);
        return LT_ERR_CUDA;
    }
    return LT_OK;
}

template <int NT, int MA>
static int launch_tc(const void* W, int ldw, const void* X, int ldx, GemmP P, cudaStream_t s) {
    using C = GemmCfg<NT, MA>;
    CUtensorMap tmW, tmX;
    int rc = make_map_bf16(&tmW, W, (long)P.M * MA, P.K, ldw, 128);
    if (rc != LT_OK) return rc;
    rc = make_map_bf16(&tmX, X, P.T, P.K, ldx, NT);
    if (rc != LT_OK) return rc;
    static PerDeviceOnce once;
    if (once.first())
        LT_CUDA(cudaFuncSetAttribute(k_gemm_tc<NT, MA>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
    P.row_tiles = (P.M + 127) / 128;
    P.t_tiles = (P.T + NT - 1) / NT;
    P.up_row = P.M;
    P.status = device_status_ptr();
    LT_REQUIRE(P.status != nullptr, "lt_dn_linear: status word unavailable");
    const long tiles = (long)P.row_tiles * P.t_tiles;
    const int sms = sm_count();
    k_gemm_tc<NT, MA><<<(int)(tiles < sms ? tiles : sms), C::THREADS, C::SMEM, s>>>(tmW, tmX, P);
    return check_launch("lt_dn_linear");
}

// ---------------------------------------------------------------------------- fp32

// ---- fp32: every product and sum an fp32 fused multiply-add on the CUDA cores, bound by the operand reads (shared memory 76
// to 79 % busy, issue slots 70 %, FMA pipe 48 %).  64 weight rows x 8 MQ
// tokens per CTA of 128 threads, a thread owns 4 rows (pairs of rows with GLU) x MQ tokens: 4 + MQ 16-byte reads of shared
// memory per 16 MQ multiply-adds, three stages of 32 k filled by asynchronous copies.  k is summed in up to four contiguous
// parts, added in order.  One CTA folds them in turn, or a cluster of as many CTAs takes one each and adds them through
// distributed shared memory: a prompt of a few hundred tokens has fewer tiles than the GPU has places for CTAs.  The bits
// are the same in every form, so a token's output does not depend on how many others share its pass.
// Against 4 x 4 per thread from single floats of one unbuffered stage, one chain over k (M x K x T): 896 x 6656 x 300
// 780 -> 113 us, 3640 x 896 x 300 117 -> 68, 8192 x 2048 x 512 gated 1075 -> 792, 896 x 6656 x 45 800 -> 49.  Shorter chains of
// sums: errors against 64 bits about half.
constexpr int F32_THREADS = 128, F32_BM = 64, F32_BK = 32, F32_ST = F32_BK + 4, F32_STAGES = 3;

template <bool GLU, int MQ, bool SHARED>
struct F32Cfg {
    static constexpr int NG = GLU ? 2 : 1, BN = 8 * MQ, ROWS = NG * F32_BM + BN;
    static constexpr int SMEM = F32_STAGES * ROWS * F32_ST * 4;
    // quads of k in flight (unrolled): as many as the registers of the resident CTAs leave room for, measured
    static constexpr int QUADS = MQ == 4 && !SHARED ? 8 : (!GLU && (MQ == 4 || !SHARED) ? 4 : 2);
    static_assert(SMEM >= NG * 4 * MQ * F32_THREADS * 4, "the partials fit the stages");
};

__device__ __forceinline__ void f32_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <bool GLU, int MQ, bool SHARED>      // SHARED: a CTA per part of k, parts of them in a cluster; else a CTA folds all
__global__ void __launch_bounds__(F32_THREADS)
k_gemm_f32(const float* __restrict__ W, int ldw, const float* __restrict__ X, int ldx, int parts, const __grid_constant__ GemmP P) {
    using C = F32Cfg<GLU, MQ, SHARED>;
    constexpr int NG = C::NG, BN = C::BN;
    extern __shared__ __align__(16) float f32_smem[];
    const int tid = threadIdx.x, n = tid & 15, m = tid >> 4;
    const int n0 = blockIdx.x * F32_BM, t0 = blockIdx.y * BN, rank = SHARED ? blockIdx.z : 0;
    const int nk = (P.K + F32_BK - 1) / F32_BK;
    auto part_from = [&](int part) { return (int)((long)nk * part / parts); };     // first chunk of a part
    const int c0 = SHARED ? part_from(rank) : 0, c1 = SHARED ? part_from(rank + 1) : nk;

    auto copy = [&](int c, int stage) {
        float* dst = f32_smem + stage * C::ROWS * F32_ST;
        if (c < c1) {
#pragma unroll
            for (int e = tid; e < C::ROWS * (F32_BK / 4); e += F32_THREADS) {
                const int r = e >> 3, k = c * F32_BK + (e & 7) * 4;          // K is a multiple of 4
                const float* src;
                bool ok = k < P.K;
                if (r < NG * F32_BM) {
                    const int row = n0 + (r & (F32_BM - 1));
                    ok = ok && row < P.M;
                    src = W + (long)((r / F32_BM) * P.up_row + row) * ldw + k;
                } else {
                    const int t = t0 + r - NG * F32_BM;
                    ok = ok && t < P.T;
                    src = X + (long)t * ldx + k;
                }
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + r * F32_ST + (e & 7) * 4)),
                             "l"(ok ? src : W), "r"(ok ? 16 : 0)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float acc[NG][MQ][4];
#pragma unroll
    for (int g = 0; g < NG; g++)
#pragma unroll
        for (int i = 0; i < MQ; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[g][i][j] = 0.0f;
#pragma unroll
    for (int s = 0; s < F32_STAGES - 1; s++) copy(c0 + s, s);
    int stage = 0, part = 0, part_end = part_from(1);
    // sums of the parts before this one wait in local memory: in registers they would halve the CTAs of an SM (zero, unknown
    // to the compiler, keeps them there)
    float before[SHARED ? 1 : NG * MQ * 4];
    int zero = 0;
    if (!SHARED) asm volatile("mov.u32 %0, 0;" : "=r"(zero));
    auto add_before = [&]() {
#pragma unroll
        for (int g = 0; g < NG; g++)
#pragma unroll
            for (int i = 0; i < MQ; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[g][i][j] = before[SHARED ? 0 : (g * MQ + i) * 4 + j + zero] + acc[g][i][j];
    };
    for (int c = c0; c < c1; c++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(F32_STAGES - 2) : "memory");
        __syncthreads();                                   // chunk c is there, chunk c - 1 is used up
        copy(c + F32_STAGES - 1, stage == 0 ? F32_STAGES - 1 : stage - 1);
        const float4* w4 = (const float4*)(f32_smem + (stage * C::ROWS + n) * F32_ST);
        const float4* x4 = (const float4*)(f32_smem + (stage * C::ROWS + NG * F32_BM + m * MQ) * F32_ST);
#pragma unroll C::QUADS
        for (int k = 0; k < F32_BK / 4; k++) {
            float4 x[MQ];
#pragma unroll
            for (int i = 0; i < MQ; i++) x[i] = x4[i * (F32_ST / 4) + k];
#pragma unroll
            for (int g = 0; g < NG; g++) {
                float4 w[4];
#pragma unroll
                for (int j = 0; j < 4; j++) w[j] = w4[(g * F32_BM + 16 * j) * (F32_ST / 4) + k];
#pragma unroll
                for (int i = 0; i < MQ; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[g][i][j] = fmaf(w[j].x, x[i].x, acc[g][i][j]);
#pragma unroll
                for (int i = 0; i < MQ; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[g][i][j] = fmaf(w[j].y, x[i].y, acc[g][i][j]);
#pragma unroll
                for (int i = 0; i < MQ; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[g][i][j] = fmaf(w[j].z, x[i].z, acc[g][i][j]);
#pragma unroll
                for (int i = 0; i < MQ; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[g][i][j] = fmaf(w[j].w, x[i].w, acc[g][i][j]);
            }
        }
        stage = stage == F32_STAGES - 1 ? 0 : stage + 1;
        if (!SHARED && c + 1 == part_end) {
            if (part > 0) add_before();
            if (++part < parts) {
#pragma unroll
                for (int g = 0; g < NG; g++)
#pragma unroll
                    for (int i = 0; i < MQ; i++)
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            before[SHARED ? 0 : (g * MQ + i) * 4 + j + zero] = acc[g][i][j];
                            acc[g][i][j] = 0.0f;
                        }
                part_end = part_from(part + 1);
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (SHARED) {       // partials [g][token][row][thread]; every CTA adds up the tokens of its share
        __syncthreads();
#pragma unroll
        for (int g = 0; g < NG; g++)
#pragma unroll
            for (int i = 0; i < MQ; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) f32_smem[((g * MQ + i) * 4 + j) * F32_THREADS + tid] = acc[g][i][j];
        f32_cluster_sync();
        const unsigned mine = smem_u32(f32_smem + tid);
#pragma unroll
        for (int i = 0; i < MQ; i++) {
            if (i * parts / MQ != rank) continue;
#pragma unroll
            for (int g = 0; g < NG; g++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    float v = 0.0f;
                    for (int r = 0; r < parts; r++) {
                        unsigned a;
                        float part;
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                                     : "=r"(a)
                                     : "r"(mine + (unsigned)(((g * MQ + i) * 4 + j) * F32_THREADS * 4)), "r"(r));
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(part) : "r"(a) : "memory");
                        v = r == 0 ? part : v + part;
                    }
                    acc[g][i][j] = v;
                }
        }
        f32_cluster_sync();     // no CTA leaves while another reads its partials
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int row = n0 + n + 16 * j;
        if (row >= P.M) continue;
        const RowEpi re = row_epi(P.epi, row);
#pragma unroll
        for (int i = 0; i < MQ; i++) {
            const int t = t0 + m * MQ + i;
            if (t >= P.T || (SHARED && i * parts / MQ != rank)) continue;
            if (GLU) glu_store<float>(P.epi, P.Y, (long)t * P.ldy + row, acc[0][i][j], acc[NG - 1][i][j]);
            else epi_store<float>(P.epi, re, P.Y, t, P.ldy, row, acc[0][i][j]);
        }
    }
}

// Parts of k that every output is added up from: of K alone, so that a token's bits do not depend on the pass it is in.
static int f32_parts(int K) { return K >= 32 * 32 ? 4 : (K >= 16 * 32 ? 2 : 1); }

template <bool GLU, int MQ, bool SHARED>
static int launch_f32(const void* W, int ldw, const void* X, int ldx, const GemmP& P, cudaStream_t s) {
    using C = F32Cfg<GLU, MQ, SHARED>;
    static PerDeviceOnce once;
    if (once.first()) LT_CUDA(cudaFuncSetAttribute(k_gemm_f32<GLU, MQ, SHARED>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
    const long gx = (P.M + F32_BM - 1) / F32_BM, gy = (P.T + C::BN - 1) / C::BN;
    LT_REQUIRE(gy <= 65535, "lt_dn_linear: T=%d too large", P.T);
    const int parts = f32_parts(P.K), S = SHARED ? parts : 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)gx, (unsigned)gy, (unsigned)S);
    cfg.blockDim = dim3(F32_THREADS);
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = (unsigned)S;
    cfg.attrs = at;
    cfg.numAttrs = SHARED ? 1 : 0;
    return check_launch("lt_dn_linear", 1,
                        cudaLaunchKernelEx(&cfg, k_gemm_f32<GLU, MQ, SHARED>, (const float*)W, ldw, (const float*)X, ldx, parts, P));
}

// The form with the least estimated time.  n CTAs together on an SM take a + b n us per chunk of 32 k each, and every round of
// them o us beside that (first loads, epilogue, exchange between the CTAs of a cluster): fitted to 223 sizes (16 matrices from
// 32 x 896 to 16384 x 1024, 2 to 2000 tokens), where the form chosen is 0.4 % off the fastest on average, 10 % at most.
// Clusters lose another 8 % where they need several rounds, since a place for one is free only when all of its CTAs find one.
// 896 x 6656, 2 tokens: 176 us with 32 tokens per CTA, 46 with k shared; 16384 x 1024, 1000 tokens: 903, 1095 and with 64
// tokens per CTA 830, shared 1300; 2048 x 8192, 1000 tokens: 920, 960, 915, 879.
struct F32Time { double a, b, o; };
template <bool GLU, int MQ, bool SHARED>
static double f32_time(const GemmP& P, const F32Time& t) {
    using C = F32Cfg<GLU, MQ, SHARED>;
    const int parts = f32_parts(P.K);
    if ((SHARED && parts == 1) || ((long)P.T + C::BN - 1) / C::BN > 65535) return 1e30;
    const int S = SHARED ? parts : 1, chunks = ((P.K + F32_BK - 1) / F32_BK + S - 1) / S;
    const long ctas = (long)((P.M + F32_BM - 1) / F32_BM) * ((P.T + C::BN - 1) / C::BN) * S;
    const long per_sm = (ctas + sm_count() - 1) / sm_count();
    const int together = 227 * 1024 / (C::SMEM + 1024);
    const long rounds = per_sm / together, rest = per_sm % together;
    double us = (double)rounds * (chunks * (t.a + t.b * together) + t.o);
    if (rest > 0) us += chunks * (t.a + t.b * (double)rest) + t.o;
    return SHARED && per_sm > together ? 1.08 * us : us;
}
template <bool GLU>
static int pick_f32(const void* W, int ldw, const void* X, int ldx, const GemmP& P, cudaStream_t s) {
    const double us[4] = {f32_time<GLU, 4, false>(P, GLU ? F32Time{0.54, 0.70, 3.0} : F32Time{0.40, 0.43, 3.0}),
                          f32_time<GLU, 4, true>(P, GLU ? F32Time{0.43, 0.81, 7.0} : F32Time{0.30, 0.46, 5.0}),
                          f32_time<GLU, 8, false>(P, GLU ? F32Time{0.45, 1.50, 7.0} : F32Time{0.30, 0.84, 9.0}),
                          f32_time<GLU, 8, true>(P, GLU ? F32Time{0.32, 1.60, 19.0} : F32Time{0.20, 0.95, 14.0})};
    int form = 0;
    for (int i = 1; i < 4; i++)
        if (us[i] < us[form]) form = i;
    if (form == 0) return launch_f32<GLU, 4, false>(W, ldw, X, ldx, P, s);
    if (form == 1) return launch_f32<GLU, 4, true>(W, ldw, X, ldx, P, s);
    if (form == 2) return launch_f32<GLU, 8, false>(W, ldw, X, ldx, P, s);
    return launch_f32<GLU, 8, true>(W, ldw, X, ldx, P, s);
}

// tile width: fewest (waves x time of a tile); a tile costs its columns plus what does not shrink with them
static int choose_nt(int M, int T, bool glu) {
    const int sms = sm_count();
    const int cand[4] = {256, 128, 64, 32};
    int best = 32;
    double cost = 1e30;
    for (int i = glu ? 1 : 0; i < 4; i++) {
        const long tiles = (long)((M + 127) / 128) * ((T + cand[i] - 1) / cand[i]);
        const double c = (double)((tiles + sms - 1) / sms) * ((glu ? 2 : 1) * cand[i] + 48);
        if (c < cost) {
            cost = c;
            best = cand[i];
        }
    }
    return best;
}

}  // namespace dn
}  // namespace lt

using namespace lt;
using namespace lt::dn;

extern "C" int lt_dn_linear(const void* W, int ldw, const void* X, int ldx, void* Y, int ldy, int f32, int M, int K, int T,
                            const lt_dn_epilogue* h_epi, int variant, void* stream) {
    LT_REQUIRE(W && X && Y, "lt_dn_linear: null pointer");
    const char* bad = epi_error(h_epi);
    LT_REQUIRE(bad == nullptr, "lt_dn_linear: %s", bad);
    LT_REQUIRE(M > 0 && T > 0 && K > 0 && K % 8 == 0, "lt_dn_linear: M=%d T=%d K=%d (K a multiple of 8)", M, T, K);
    LT_REQUIRE(ldw >= K && ldw % 8 == 0 && ldx >= K && ldx % 8 == 0, "lt_dn_linear: ldw=%d ldx=%d must be multiples of 8, >= K=%d",
               ldw, ldx, K);
    const int my = h_epi->kind == LT_DN_STORE && h_epi->tail != nullptr && h_epi->tail_from < M ? h_epi->tail_from : M;
    LT_REQUIRE(ldy >= my, "lt_dn_linear: ldy=%d < M=%d", ldy, my);
    LT_REQUIRE(h_epi->kind != LT_DN_STORE_GLU, "lt_dn_linear: the combined epilogue is lt_dn_gemv's");
    LT_REQUIRE(aligned16(W) && aligned16(X), "lt_dn_linear: W and X must be 16-byte aligned");
    LT_REQUIRE(variant == 0 || variant == 32 || variant == 64 || variant == 128 || variant == 256,
               "lt_dn_linear: unknown variant %d", variant);
    cudaStream_t s = (cudaStream_t)stream;
    GemmP P = {};
    P.Y = Y; P.M = M; P.K = K; P.T = T; P.ldy = ldy; P.epi = *h_epi; P.up_row = M;
    const bool glu = h_epi->kind == LT_DN_GLU;
    if (f32)
        return glu ? pick_f32<true>(W, ldw, X, ldx, P, s) : pick_f32<false>(W, ldw, X, ldx, P, s);
    const int nt = variant ? variant : choose_nt(M, T, glu);
    if (glu) {
        LT_REQUIRE(nt <= 128, "lt_dn_linear: tiles of 256 tokens do not fit a gated pair");
        if (nt == 128) return launch_tc<128, 2>(W, ldw, X, ldx, P, s);
        if (nt == 64) return launch_tc<64, 2>(W, ldw, X, ldx, P, s);
        return launch_tc<32, 2>(W, ldw, X, ldx, P, s);
    }
    if (nt == 256) return launch_tc<256, 1>(W, ldw, X, ldx, P, s);
    if (nt == 128) return launch_tc<128, 1>(W, ldw, X, ldx, P, s);
    if (nt == 64) return launch_tc<64, 1>(W, ldw, X, ldx, P, s);
    return launch_tc<32, 1>(W, ldw, X, ldx, P, s);
}
