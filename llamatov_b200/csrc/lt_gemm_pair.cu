// Q8_0 GEMM on the tensor cores, block sums AND block scales (tcgen05, kind::i8 and kind::f16).
//
// The arithmetic contract is lt_gemm_tc.cu's.  Per output and block it asks for one product of scales, one conversion of the
// integer sum and one multiply-add; this kernel leaves only the last two to the CUDA cores:
//   S[n, t] = f32(Wd[n, b]) * f32(Xd[t, b]) is a product of two fp16 numbers, exact in fp32 (22 bits), so a second MMA with
//   one non-zero k per block makes the same bits as __fmul_rn (all pairs of exponents, subnormals too).  Its operands are the
//   scales themselves, without conversion: A[n, k] = Wd[n, b_k], B[(k, t), k'] = Xd[t, b_k] where k' = k, else 0.
// Zeros next to a weight scale that is not finite turn NaN; rows that hold one are made anew from global memory (`repair`).
//
// A stage is two blocks b and b + 16 (lanes l and l + 16 of the contract, l < 16, b = l + 32 r): their tree level s = 16 is
// the first addition, so an output needs two running sums and four waiting subtrees instead of the sixteen registers of chunks
// of adjacent blocks, and a CTA's tile can be 128 rows x 32 columns.  l is visited in bit-reversed order, r ascending.
//
// What bounded the 16-column tiles (9728 x 896 x 2048, 264 us): 1070 clocks per 8192 block sums, of which 256 are shared-memory
// reads of activation scales (a broadcast 16-byte read still writes 512 bytes of registers), the rest uncoalesced loads of
// weight scales and hand-overs.  Here 480 clocks (139 us; 28672 x 4096 x 512 683 -> 379 us, 4096 x 14336 x 512 330 -> 228 us):
// the epilogue's issue slots, 68 to 70 % busy by the counters; by count, conversions and fp32 pipes have 128 of the 480 to do, the MMAs 130.
// An epilogue thread is one row x 16 columns; a copy of its sums or a poll costs as much as a fold, and its waits are as long
// as its arithmetic, so two sets of eight epilogue warps work on different l (the even and the odd ones).
// Two kernels: k_q8_gemm_res for rows of 512 to 896 values, k_q8_gemm_pair for any; lt_q8_gemm_tc chooses between them and the
// 16-column tiles by time.  Every wait is bounded, as in lt_gemm_tc.cu.
#include <stddef.h>

#include "lt_gemm_pair.cuh"
#include "lt_tc.cuh"

namespace lt {
namespace tc {
namespace pair {

constexpr int TM = 128, NT = 32, CW = 16, EW = 8;       // EW: epilogue warps of a set
constexpr int NSLOT = 4, SLOT_COLS = 4 * NT;            // a slot: sums of two blocks, then their scales
constexpr int W_BLOCK = TM * 32, X_BLOCK = NT * 32;     // bytes of one block of a tile

struct Params {
    const unsigned short *Wd, *Xd;
    const signed char *Wq, *Xq;
    const float* Resid;
    float* Y;
    int* status;
    int M, K, T;
    int col_tiles, units;   // units = row tiles x column tiles
    int resid_ld;
};

__device__ __forceinline__ void mma_f16(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc)
        : "memory");
}
// K-major operand without swizzle: rows of 16 bytes, 8-row groups 128 bytes apart, the second 16 bytes of k `lbo` bytes further
__device__ __forceinline__ unsigned long long plain_desc(unsigned addr, unsigned lbo) {
    return (unsigned long long)((addr >> 4) & 0x3FFFu) | ((unsigned long long)(lbo >> 4) << 16) | ((unsigned long long)(128 >> 4) << 32) |
           (1ull << 46);
}
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// 8 columns of sums at `a` and of scales at `b`, with the wait in the same statement: registers handed through a statement of
// their own after the wait cost a move each (a third of the epilogue's instructions)
__device__ __forceinline__ void tmem_ld_pair(unsigned a, unsigned b, int (&v)[8], int (&s)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%16];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%17];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(s[0]), "=r"(s[1]),
          "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7])
        : "r"(a), "r"(b)
        : "memory");
}

// y: the N outputs of this lane's row, from column `first` on, before the residual.  Zeros beside a weight scale that is not finite
// make NaNs of their block's neighbours in the scale operand, but such a scale leaves no finite output in its row either way
// (infinity times a sum, or times zero), so a row that has one is recognised by an output that is not finite.  A warp then looks
// through the row's scales (others may be so by their activations) and makes its outputs by the contract alone, lane = lane:
// 4096 x 14336 x 256 with one such row in 128: 168 us (110 without; one thread byte by byte 12280).
template <int N, int L>
__device__ __forceinline__ void repair(const Params& P, int row, int first, int valid, float (&y)[L]) {
    bool odd = false;
#pragma unroll
    for (int c = 0; c < N; c++) odd |= c < valid && (__float_as_uint(y[c]) & 0x7F800000u) == 0x7F800000u;
    unsigned todo = __ballot_sync(0xffffffffu, odd && row < P.M);
    const int lane = threadIdx.x & 31, nb = P.K >> 5;
#pragma unroll 1
    for (; todo != 0; todo &= todo - 1) {
        const int src = __ffs(todo) - 1, r = __shfl_sync(0xffffffffu, row, src);
        const unsigned short* wd = P.Wd + (long)r * nb;
        bool bad = false;
#pragma unroll 4
        for (int b = lane; b < nb; b += 32) bad |= (wd[b] & 0x7C00) == 0x7C00;
        if (!__any_sync(0xffffffffu, bad)) continue;
#pragma unroll 1
        for (int c = 0; c < N && c < valid; c++) {
            const unsigned short* xd = P.Xd + (long)(first + c) * nb;
            const int4 *w4 = (const int4*)(P.Wq + (long)r * P.K), *x4 = (const int4*)(P.Xq + (long)(first + c) * P.K);
            float acc = 0.0f;
#pragma unroll 1
            for (int b = lane; b < nb; b += 32) {
                const int4 w0 = __ldg(w4 + 2 * b), w1 = __ldg(w4 + 2 * b + 1), x0 = __ldg(x4 + 2 * b), x1 = __ldg(x4 + 2 * b + 1);
                int sum = __dp4a(w0.x, x0.x, __dp4a(w0.y, x0.y, __dp4a(w0.z, x0.z, __dp4a(w0.w, x0.w, 0))));
                sum = __dp4a(w1.x, x1.x, __dp4a(w1.y, x1.y, __dp4a(w1.z, x1.z, __dp4a(w1.w, x1.w, sum))));
                const float s = __fmul_rn(__half2float(__ushort_as_half(wd[b])), __half2float(__ushort_as_half(xd[b])));
                acc = __fmaf_rn(s, (float)sum, acc);
            }
            acc = __shfl_sync(0xffffffffu, warp_tree_sum(acc), 0);
#pragma unroll
            for (int k = 0; k < N; k++)
                if (k == c && lane == src) y[k] = acc;
        }
    }
}

// ---------------------------------------------------------------------------- rows of at most 896 values

// Every lane has at most one block, so a tile is sixteen stages of blocks l and l + 16, the weights of a row tile (at most
// 128 KB) stay in shared memory while the CTA goes through column tiles, and every loop over stages is unrolled.  Weights come
// as boxes of one block (32 bytes a row), each as soon as the last tile has passed its place; activations as whole tiles, two
// ahead; scale operands by halves of a tile (the even l, then the odd l).  Weight scales are packed 8 to a row of 16 bytes
// (four stages); which of them a stage means is in its activation operand, whose other places are zero.
// Two sets of eight epilogue warps and two MMA warps: set h folds the even (0) or the odd (1) l of every tile, from two slots
// of its own, and the sets exchange half of their columns for the last level, s = 1.
constexpr int RES_THREADS = (2 * EW + 4) * 32;
constexpr int RES_EPI_REGS = 104, RES_AUX_REGS = 64;     // (512 x 104 + 128 x 64) registers are what 640 threads of 96 start with
enum : unsigned {             // byte offsets of the barriers
    R_WFULL = 0, R_XFULL = 128, R_XEMPTY = 144, R_SFULL = 160, R_SEMPTY = 176, R_TFULL = 192, R_TEMPTY = 224
};
struct ResBars {
    unsigned long long wfull[16], xfull[2], xempty[2], sfull[2], sempty[2], tfull[NSLOT], tempty[NSLOT];
    unsigned tmem_base;
    int abort_flag;
};
static_assert(offsetof(ResBars, xfull) == R_XFULL && offsetof(ResBars, sempty) == R_SEMPTY && offsetof(ResBars, tempty) == R_TEMPTY,
              "offsets");
constexpr int RES_A = 4 * TM * 16, RES_B_STAGE = 2 * NT * 16, RES_B = 16 * RES_B_STAGE, RES_ZERO = TM * 16;
constexpr int RES_MAX_K = 896;    // what 227 KB hold
struct ResSmem {   // byte offsets from a 1024-byte boundary
    int x, a, b, zero, bars, xchg, total;
    __host__ __device__ explicit ResSmem(int nb)
        : x(nb * W_BLOCK), a(x + 2 * nb * X_BLOCK), b(a + RES_A), zero(b + RES_B), bars(zero + RES_ZERO), xchg(bars + 512),
          total(xchg + TM * NT * 4) {}
};
static_assert(sizeof(ResBars) <= 512, "barriers");

__device__ __forceinline__ constexpr int brev4(int q) { return (q & 1) << 3 | (q & 2) << 1 | (q & 4) >> 1 | (q & 8) >> 3; }

__global__ void __launch_bounds__(RES_THREADS, 1)
k_q8_gemm_res(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const Params P) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int nb = P.K >> 5;
    const ResSmem L(nb);
    ResBars* B = (ResBars*)(base + L.bars);
    float* xchg = (float*)(base + L.xchg);
    const unsigned sb = smem_u32(base), bars = sb + (unsigned)L.bars;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int u0 = (int)((long)P.units * blockIdx.x / gridDim.x), u1 = (int)((long)P.units * (blockIdx.x + 1) / gridDim.x);
    volatile int* abort_flag = &B->abort_flag;

    for (int i = tid; i < (L.bars - L.a) / 16; i += RES_THREADS) ((uint4*)(base + L.a))[i] = make_uint4(0u, 0u, 0u, 0u);
    if (warp == 0) {
        if (lane < 16) mbar_init(&B->wfull[lane], 1);
        if (lane < 2) {
            mbar_init(&B->xfull[lane], 1);
            mbar_init(&B->xempty[lane], 2);
            mbar_init(&B->sfull[lane], 1);
            mbar_init(&B->sempty[lane], 1);
        }
        if (lane < NSLOT) {
            mbar_init(&B->tfull[lane], 1);
            mbar_init(&B->tempty[lane], EW);
        }
        if (lane == 0) B->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 2 * EW + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&B->tmem_base)),
                     "r"((unsigned)(NSLOT * SLOT_COLS))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = __shfl_sync(0xffffffffu, B->tmem_base, 0);   // uniform, as the loads want it

    // f(row tile, column tile, its number in this CTA, whether the row tile is new)
    auto tiles = [&](auto f) {
        if (u0 >= u1) return;
        int rt = u0 / P.col_tiles, tt = u0 - rt * P.col_tiles;
        bool fresh = true;
#pragma unroll 1
        for (int n = 0; n < u1 - u0; n++) {
            f(rt, tt, n, fresh);
            fresh = ++tt == P.col_tiles;
            if (fresh) {
                tt = 0;
                rt++;
            }
        }
    };
    auto wait = [&](unsigned bar, unsigned parity) { bar_wait(bar_test(bar, parity), bar, parity, abort_flag, P.status); };

    if (warp >= 2 * EW) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(RES_AUX_REGS));
        if (warp == 2 * EW) {
            // -------------------------------------------------------------- TMA
            const bool one = elect_one();
            tiles([&](int rt, int tt, int n, bool fresh) {
                const unsigned buf = n & 1, xf = bars + R_XFULL + 8 * buf;
                if (!acquire(bars + R_XEMPTY + 8 * buf, ((n >> 1) & 1) ^ 1, abort_flag, P.status)) return;
                if (one) bar_expect_tx(xf, nb * X_BLOCK);
                if (one)
                    for (int c = 0; c < nb / 4; c++) tma_load_2d(sb + L.x + (buf * nb + 4 * c) * X_BLOCK, &tmX, c * 128, tt * NT, xf);
                if (fresh) {
                    // the places of a half are free when the last tile's MMAs of that half are complete
#pragma unroll 1
                    for (int q = 0; q < 16; q++) {
                        if ((q & 7) == 0 && !acquire(bars + R_SEMPTY + q, (n & 1) ^ 1, abort_flag, P.status)) return;
                        const int l = brev4(q), two = l + 16 < nb;
                        const unsigned wf = bars + R_WFULL + 8 * q;
                        if (one) {
                            bar_expect_tx(wf, (1 + two) * W_BLOCK);
                            tma_load_2d(sb + l * W_BLOCK, &tmW, l * 32, rt * TM, wf);
                        }
                        if (one && two) tma_load_2d(sb + (l + 16) * W_BLOCK, &tmW, l * 32 + 512, rt * TM, wf);
                    }
                }
            });
        } else if (warp <= 2 * EW + 2) {
            const bool one = elect_one();
            // -------------------------------------------------------------- MMA
            constexpr unsigned idesc_i8 = (2u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(NT >> 3) << 17) | ((unsigned)(TM >> 4) << 24);
            constexpr unsigned idesc_f16 = (1u << 4) | ((unsigned)(2 * NT >> 3) << 17) | ((unsigned)(TM >> 4) << 24);
            const unsigned long long wdesc = smem_desc<1>(sb);
            const unsigned long long adesc = plain_desc(sb + L.a, L.zero - L.a), bdesc = plain_desc(sb + L.b, L.zero - L.b);
            // a step of an operand's place: its address up, the distance to the zeros down (16-byte units)
            constexpr unsigned long long astep = (TM * 16 >> 4) - ((unsigned long long)(TM * 16 >> 4) << 16);
            constexpr unsigned long long bstep = (RES_B_STAGE >> 4) - ((unsigned long long)(RES_B_STAGE >> 4) << 16);
            const int h = warp - (2 * EW + 1);
            unsigned rows = 0;   // row tiles begun
            bool free_slot = true;   // the answer for the next stage's slot
            tiles([&](int, int, int n, bool fresh) {
                const unsigned long long xdesc = smem_desc<4>(sb + L.x + (n & 1) * nb * X_BLOCK);
                rows += fresh;
                wait(bars + R_XFULL + 8 * (n & 1), (n >> 1) & 1);
                wait(bars + R_SFULL + 8 * h, n & 1);
#pragma unroll 1
                for (int j = 0; j < 8; j++) {
                    const int q = 8 * h + j, l = brev4(j) + h;
                    const unsigned slot = 2 * h + (j & 1), d = tmem + slot * SLOT_COLS;
                    if (fresh) wait(bars + R_WFULL + 8 * q, (rows & 1) ^ 1);
                    bar_wait(free_slot, bars + R_TEMPTY + 8 * slot, ((j >> 1) & 1) ^ 1, abort_flag, P.status);
                    const int jn = (j + 1) & 7;
                    free_slot = bar_test(bars + R_TEMPTY + 8 * (2 * h + (jn & 1)), ((jn >> 1) & 1) ^ 1);
                    tc_fence_after();
                    // block b of the activations: 32 bytes of the 128-byte rows of chunk b / 4
                    const unsigned long long wd = wdesc + l * (W_BLOCK >> 4), xd = xdesc + (l >> 2) * (4 * X_BLOCK >> 4) + (l & 3) * 2;
                    if (one) {
                        mma_i8(d, wd, xd, idesc_i8);
                        mma_f16(d + 2 * NT, adesc + (q / 4) * astep, bdesc + q * bstep, idesc_f16);
                        if (l + 16 < nb) mma_i8(d + NT, wd + 16 * (W_BLOCK >> 4), xd + 4 * (4 * X_BLOCK >> 4), idesc_i8);
                        bar_commit(bars + R_TFULL + 8 * slot);
                    }
                }
                if (one) {
                    bar_commit(bars + R_SEMPTY + 8 * h);
                    bar_commit(bars + R_XEMPTY + 8 * (n & 1));
                }
            });
        } else {
            // -------------------------------------------------------------- scales
            // Lane = a row.  w[k] holds the scales of blocks 2 k and 2 k + 1: the low halves of w[k] and w[k + 8] are a stage of
            // half 0 (l = 2 k), the high halves one of half 1.
            const bool vec = ((((uintptr_t)P.Wd) | ((uintptr_t)P.Xd)) & 7) == 0;
            auto fetch = [&](const unsigned short* p, unsigned (&w)[16]) {
#pragma unroll
                for (int k = 0; k < 16; k += 2) {
                    uint2 u = make_uint2(0u, 0u);
                    if (2 * k < nb) {
                        if (vec) u = __ldg((const uint2*)(p + 2 * k));
                        else u = make_uint2(__ldg(p + 2 * k) | (unsigned)__ldg(p + 2 * k + 1) << 16,
                                            __ldg(p + 2 * k + 2) | (unsigned)__ldg(p + 2 * k + 3) << 16);
                    }
                    w[k] = u.x;
                    w[k + 1] = u.y;
                }
            };
            tiles([&](int rt, int tt, int n, bool fresh) {
                const int t = tt * NT + lane;
                unsigned x[16];
                fetch(P.Xd + (long)(t < P.T ? t : P.T - 1) * nb, x);
                if (fresh) {
                    wait(bars + R_SEMPTY, (n & 1) ^ 1);
                    wait(bars + R_SEMPTY + 8, (n & 1) ^ 1);
                    unsigned w[2][16];
                    auto row_of = [&](int r) {   // rows past the end read the last row's scales; nothing of them is stored
                        const int row = rt * TM + r;
                        return P.Wd + (long)(row < P.M ? row : P.M - 1) * nb;
                    };
                    fetch(row_of(lane), w[0]);
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        if (r < 3) fetch(row_of(lane + 32 * (r + 1)), w[(r + 1) & 1]);
                        const unsigned(&c)[16] = w[r & 1];
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const unsigned sel = h ? 0x7632u : 0x5410u;
                            uint4* ap = (uint4*)(base + L.a + h * 2 * TM * 16 + (lane + 32 * r) * 16);
                            auto pick = [&](int k) { return __byte_perm(c[k], c[k + 8], sel); };
                            ap[0] = make_uint4(pick(0), pick(4), pick(2), pick(6));
                            ap[TM] = make_uint4(pick(1), pick(5), pick(3), pick(7));
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    wait(bars + R_SEMPTY + 8 * h, (n & 1) ^ 1);
                    unsigned char* bp = base + L.b + h * 8 * RES_B_STAGE + lane * 16;
#pragma unroll
                    for (int j = 0; j < 8; j++) {   // stage 8 h + j is l = 2 k + h
                        const int k = brev4(j) >> 1;
                        *(unsigned short*)(bp + j * RES_B_STAGE + (j & 3) * 4) = (unsigned short)(x[k] >> (16 * h));
                        *(unsigned short*)(bp + j * RES_B_STAGE + NT * 16 + (j & 3) * 4 + 2) = (unsigned short)(x[k + 8] >> (16 * h));
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) bar_arrive(bars + R_SFULL + 8 * h);
                }
            });
        }
    } else {
        // ------------------------------------------------------------------ epilogue
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(RES_EPI_REGS));
        const int qr = warp & 3, cg = (warp >> 2) & 1, h = warp >> 3, col0 = cg * CW;
        const unsigned taddr0 = tmem + ((unsigned)(qr * 32) << 16) + (unsigned)(col0 + 2 * h * SLOT_COLS);
        const unsigned tfull = bars + R_TFULL + 16 * h, tempty = bars + R_TEMPTY + 16 * h;
        int v[8], sc[8];
        auto load = [&](int slot, int j, int c8) {   // columns 8 c8 .. of block j of a slot
            const unsigned a = taddr0 + slot * SLOT_COLS + j * NT + c8 * 8;
            tmem_ld_pair(a, a + 2 * NT, v, sc);
        };
        auto product = [&](int c) {
            const f32x2 f = pack2((float)v[2 * c], (float)v[2 * c + 1]);
            return fma2(pack2(__int_as_float(sc[2 * c]), __int_as_float(sc[2 * c + 1])), f, 0ull);
        };
        bool next = false;
        tiles([&](int rt, int tt, int n, bool) {
            f32x2 st[3][CW / 2], x[CW / 2];
            // Four stages at a time: sixteen in a row do not fit the instruction caches (no_instruction was the first stall).  Every
            // stage writes where its value is wanted (146 -> 139 us at 9728 x 896 x 2048).
#pragma unroll 1
            for (int g = 0; g < 2; g++) {
                auto stage = [&](int i, f32x2 (&out)[CW / 2]) {   // stage j = 4 g + i, l = brev4(j) + h
                    const bool two = (brev4(i) | brev4(4) * g) + h + 16 < nb;
                    const int slot = i & 1, parity = (i >> 1) & 1;      // stage j's slot is used (j / 2)-th
                    bar_wait(next, tfull + 8 * slot, parity, abort_flag, P.status);
                    tc_fence_after();
#pragma unroll
                    for (int c8 = 0; c8 < 2; c8++) {
                        load(slot, 0, c8 ^ h);
#pragma unroll
                        for (int c = 0; c < 4; c++) out[4 * c8 + c] = product(c);
                    }
                    next = bar_test(tfull + 8 * (slot ^ 1), ((i + 1) >> 1) & 1);
                    if (two) {
                        load(slot, 1, h);
#pragma unroll
                        for (int c = 0; c < 4; c++) out[c] = add2(out[c], product(c));
                        load(slot, 1, 1 ^ h);
                    }
                    tc_fence_before();
                    __syncwarp();
                    bar_arrive_if(lane == 0, tempty + 8 * slot);
                    if (two) {
#pragma unroll
                        for (int c = 0; c < 4; c++) out[4 + c] = add2(out[4 + c], product(c));
                    } else {
#pragma unroll
                        for (int c = 0; c < CW / 2; c++) out[c] = add2(out[c], 0ull);
                    }
                };
                auto join = [&](f32x2 (&left)[CW / 2], f32x2 (&right)[CW / 2], f32x2 (&out)[CW / 2]) {
#pragma unroll
                    for (int c = 0; c < CW / 2; c++) out[c] = add2(left[c], right[c]);
                };
                stage(0, st[0]);
                stage(1, x);
                join(st[0], x, st[1]);
                stage(2, st[0]);
                stage(3, x);
                join(st[0], x, x);
                if (g == 0) join(st[1], x, st[2]);
                else join(st[1], x, x);
            }
#pragma unroll
            for (int c = 0; c < CW / 2; c++) x[c] = add2(st[2][c], x[c]);
            // the last level: this set finishes the columns 8 h .. 8 h + 7 of each group of 16, which are its first four pairs
            float y[CW];
#pragma unroll
            for (int c = 0; c < CW / 2; c++) unpack2(x[c], y[2 * c], y[2 * c + 1]);
            const int r = qr * 32 + lane, row = rt * TM + r;
            float* xp = xchg + (cg * 16) * TM + r;      // [group][set that finishes][8][row]
            if (n > 0) asm volatile("bar.sync 1, %0;" ::"n"(2 * EW * 32) : "memory");   // the last tile's partials have been read
#pragma unroll
            for (int c = 0; c < 8; c++) xp[((1 - h) * 8 + c) * TM] = y[8 + c];
            asm volatile("bar.sync 2, %0;" ::"n"(2 * EW * 32) : "memory");
            const int first = tt * NT + col0 + 8 * h, valid = P.T - first;
#pragma unroll
            for (int c = 0; c < 8; c++) y[c] = __fadd_rn(y[c], xp[(h * 8 + c) * TM]);
            if (valid > 0) repair<8>(P, row, first, valid, y);
            if (row < P.M && valid > 0) {
                if (P.Resid != nullptr) {
                    const float* rp = P.Resid + (long)first * P.resid_ld + row;
#pragma unroll
                    for (int c = 0; c < 8; c++, rp += P.resid_ld)
                        if (c < valid) y[c] = __fadd_rn(y[c], *rp);
                }
                float* yp = P.Y + (long)first * P.M + row;
                if (valid >= 8) {
#pragma unroll
                    for (int c = 0; c < 8; c++, yp += P.M) *yp = y[c];
                } else {
#pragma unroll
                    for (int c = 0; c < 7; c++, yp += P.M)
                        if (c < valid) *yp = y[c];
                }
            }
        });
    }

    // ---------------------------------------------------------------------- teardown
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && warp == 2 * EW && lane == 0) {   // bulk copies still in flight land before the CTA leaves
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) {
        }
    }
    __syncthreads();
    if (warp == 2 * EW + 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((unsigned)(NSLOT * SLOT_COLS))
                     : "memory");
    }
}

// ---------------------------------------------------------------------------- rows of any length

// A step of the ring is four blocks b, b + 16, b + 1, b + 17 (b = l + 32 r, l even): one stage for each set, so that both stages'
// weights come in boxes 64 bytes wide (32-byte boxes are bound by the copy engine at one row a clock: 9.2 TB/s over all SMs,
// 64-byte ones bring 15.2) and both scales of a row are one word.  Blocks past the end of the rows are zeros with zero scales.
constexpr int P_NST = 6, P_LOAD = 3, P_THREADS = RES_THREADS;     // steps of the ring, warps that load
enum : unsigned { P_FULL = 0, P_EMPTY = 8 * P_NST, P_TFULL = 16 * P_NST, P_TEMPTY = P_TFULL + 32 };
struct PairBars {
    unsigned long long full[P_NST], empty[P_NST], tfull[NSLOT], tempty[NSLOT];
    unsigned tmem_base;
    int abort_flag;
};
static_assert(sizeof(PairBars) <= 512, "barriers");
struct PairSmem {   // byte offsets from a 1024-byte boundary
    static constexpr int W = 0, X = W + P_NST * 4 * W_BLOCK, A = X + P_NST * 4 * X_BLOCK, B = A + P_NST * TM * 16,
                         ZERO = B + P_NST * 4 * NT * 16, BARS = ZERO + TM * 16, XCHG = BARS + 512, TOP = XCHG + TM * NT * 4,
                         TOTAL = TOP + 2 * TM * NT * 4;
};
__device__ __forceinline__ int pair_lane(int j) { return 2 * (int)(__brev((unsigned)j) >> 29); }   // set 0's lane at visiting position j

__global__ void __launch_bounds__(P_THREADS, 1)
k_q8_gemm_pair(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const Params P) {
    using M = PairSmem;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    PairBars* B = (PairBars*)(base + M::BARS);
    float* xchg = (float*)(base + M::XCHG);
    const unsigned sb = smem_u32(base), bars = sb + M::BARS;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int nb = P.K >> 5;
    volatile int* abort_flag = &B->abort_flag;

    for (int i = tid; i < (M::BARS - M::A) / 16; i += P_THREADS) ((uint4*)(base + M::A))[i] = make_uint4(0u, 0u, 0u, 0u);
    if (warp == 0) {
        if (lane < P_NST) {
            mbar_init(&B->full[lane], 2);       // the expected bytes and the scales, both by a load warp
            mbar_init(&B->empty[lane], 1);
        }
        if (lane < NSLOT) {
            mbar_init(&B->tfull[lane], 1);
            mbar_init(&B->tempty[lane], EW);
        }
        if (lane == 0) B->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 2 * EW) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&B->tmem_base)),
                     "r"((unsigned)(NSLOT * SLOT_COLS))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = __shfl_sync(0xffffffffu, B->tmem_base, 0);

    // f(row tile, column tile) and, inside, g(set 0's block) over the steps of a tile.  Neighbours take the columns of the same
    // rows at the same time: long rows that every CTA would stream once per column tile do not fit L2 (28672 x 14336 x 48).
    auto tiles = [&](auto f) {
#pragma unroll 1
        for (int u = blockIdx.x; u < P.units; u += gridDim.x) {
            const int rt = u / P.col_tiles;
            f(rt, u - rt * P.col_tiles);
        }
    };
    auto steps = [&](auto g) {
#pragma unroll 1
        for (int j = 0; j < 8; j++)
#pragma unroll 1
            for (int b = pair_lane(j); b < nb; b += 32) g(b);
    };

    if (warp >= 2 * EW) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(RES_AUX_REGS));
        if (warp == 2 * EW) {
            // -------------------------------------------------------------- MMA
            const bool one = elect_one();
            constexpr unsigned idesc_i8 = (2u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(NT >> 3) << 17) | ((unsigned)(TM >> 4) << 24);
            constexpr unsigned idesc_f16 = (1u << 4) | ((unsigned)(2 * NT >> 3) << 17) | ((unsigned)(TM >> 4) << 24);
            // 16-byte units: the other set's block is the next 32 bytes of the 64-byte rows, the block 16 further another box
            constexpr unsigned set = 2, w16 = 2 * W_BLOCK >> 4, x16 = 2 * X_BLOCK >> 4;
            const unsigned long long wdesc = smem_desc<2>(sb + M::W), xdesc = smem_desc<2>(sb + M::X);
            const unsigned long long adesc = plain_desc(sb + M::A, M::ZERO - M::A), bdesc = plain_desc(sb + M::B, M::ZERO - M::B);
            // a step of an operand's place: its address up, the distance to the zeros down
            constexpr unsigned long long astep = (TM * 16 >> 4) - ((unsigned long long)(TM * 16 >> 4) << 16);
            constexpr unsigned long long bset = (2 * NT * 16 >> 4) - ((unsigned long long)(2 * NT * 16 >> 4) << 16), bstep = 2 * bset;
            unsigned s = 0, phase = 0, slot = 0, slot_phase = 1;
            bool ready = false, free0 = true, free1 = true;
            tiles([&](int, int) {
                steps([&](int) {
                    const unsigned d = tmem + slot * SLOT_COLS, tfull = bars + P_TFULL + 8 * slot, tempty = bars + P_TEMPTY + 8 * slot;
                    const unsigned empty = bars + P_EMPTY + 8 * s;
                    const unsigned long long wd = wdesc + s * (4 * W_BLOCK >> 4), xd = xdesc + s * (4 * X_BLOCK >> 4);
                    const unsigned long long ad = adesc + s * astep, bd = bdesc + s * bstep;
                    bar_wait(ready, bars + P_FULL + 8 * s, phase, abort_flag, P.status);
                    bar_wait(free0, tempty, slot_phase, abort_flag, P.status);
                    tc_fence_after();
                    if (one) {
                        mma_i8(d, wd, xd, idesc_i8);
                        mma_f16(d + 2 * NT, ad, bd, idesc_f16);
                        mma_i8(d + NT, wd + w16, xd + x16, idesc_i8);
                        bar_commit(tfull);
                    }
                    bar_wait(free1, tempty + 16, slot_phase, abort_flag, P.status);
                    if (++s == P_NST) {
                        s = 0;
                        phase ^= 1;
                    }
                    slot ^= 1;
                    if (slot == 0) slot_phase ^= 1;
                    ready = bar_test(bars + P_FULL + 8 * s, phase);
                    free0 = bar_test(bars + P_TEMPTY + 8 * slot, slot_phase);
                    free1 = bar_test(bars + P_TEMPTY + 8 * slot + 16, slot_phase);
                    tc_fence_after();
                    if (one) {
                        mma_i8(d + 2 * SLOT_COLS, wd + set, xd + set, idesc_i8);
                        mma_f16(d + 2 * SLOT_COLS + 2 * NT, ad, bd + bset, idesc_f16);
                        mma_i8(d + 2 * SLOT_COLS + NT, wd + set + w16, xd + set + x16, idesc_i8);
                        bar_commit(tfull + 16);
                        bar_commit(empty);
                    }
                });
            });
        } else {
            // -------------------------------------------------------------- loads, every P_LOAD-th step a warp
            // Tiles by TMA; scales through registers, requested one of this warp's steps before they are written.  28672 x 4096 x
            // 512: 576 us with one warp for the scales, 444 with two load warps, 379 with three (a single MMA warp is enough).
            // Lane = a row (and a column); the word of a row holds set 0's and set 1's scale.
            const bool one = elect_one();
            const bool words = ((((uintptr_t)P.Wd) | ((uintptr_t)P.Xd)) & 3) == 0;
            auto word = [&](const unsigned short* all, unsigned row, int b) {
                const unsigned short* p = all + (row + (unsigned)b);
                if (b >= nb) return 0u;
                return words ? __ldg((const unsigned*)p) : (unsigned)__ldg(p) | (unsigned)__ldg(p + 1) << 16;
            };
            unsigned s = (unsigned)(warp - (2 * EW + 1)), skip = s, phase = 1;
            unsigned w[4][2], x[2];
            int held_b = 0, held_row = 0, held_col = 0;
            bool any = false;
            auto write = [&]() {
                const unsigned full = bars + P_FULL + 8 * s, wdst = sb + M::W + s * 4 * W_BLOCK, xdst = sb + M::X + s * 4 * X_BLOCK;
                if (!acquire(bars + P_EMPTY + 8 * s, phase, abort_flag, P.status)) return;
                if (one) {
                    bar_expect_tx(full, 4 * (W_BLOCK + X_BLOCK));
                    tma_load_2d(wdst, &tmW, held_b * 32, held_row, full);
                    tma_load_2d(xdst, &tmX, held_b * 32, held_col, full);
                    tma_load_2d(wdst + 2 * W_BLOCK, &tmW, held_b * 32 + 512, held_row, full);
                    tma_load_2d(xdst + 2 * X_BLOCK, &tmX, held_b * 32 + 512, held_col, full);
                }
                __syncwarp();
                // A: k = 0, 1 set 0's two blocks, k = 2, 3 set 1's
#pragma unroll
                for (int j = 0; j < 4; j++)
                    *(uint2*)(base + M::A + s * TM * 16 + (lane + 32 * j) * 16) =
                        make_uint2(__byte_perm(w[j][0], w[j][1], 0x5410), __byte_perm(w[j][0], w[j][1], 0x7632));
                unsigned char* bp = base + M::B + s * 4 * NT * 16 + lane * 16;
#pragma unroll
                for (int i = 0; i < 4; i++) *(unsigned short*)(bp + i * NT * 16 + 2 * i) = (unsigned short)(x[i & 1] >> (16 * (i >> 1)));
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) bar_arrive(full);
                s += P_LOAD;
                if (s >= P_NST) {
                    s -= P_NST;
                    phase ^= 1;
                }
            };
            static_assert(P_NST % P_LOAD == 0, "a warp keeps to its places");
            tiles([&](int rt, int tt) {
                unsigned row[4];     // 32 bits of offset are enough for a matrix of 2^37 values
#pragma unroll
                for (int j = 0; j < 4; j++) {   // rows past the end read the last row's scales; nothing of them is stored
                    const int r = rt * TM + lane + 32 * j;
                    row[j] = (unsigned)(r < P.M ? r : P.M - 1) * (unsigned)nb;
                }
                const int t = tt * NT + lane;
                const unsigned xrow = (unsigned)(t < P.T ? t : P.T - 1) * (unsigned)nb;
                steps([&](int b) {
                    if (skip != 0) {
                        skip--;
                        return;
                    }
                    skip = P_LOAD - 1;
                    unsigned w1[4][2], x1[2];
#pragma unroll
                    for (int i = 0; i < 2; i++) {
#pragma unroll
                        for (int j = 0; j < 4; j++) w1[j][i] = word(P.Wd, row[j], b + 16 * i);
                        x1[i] = word(P.Xd, xrow, b + 16 * i);
                    }
                    if (any) write();
                    any = true;
                    held_b = b;
                    held_row = rt * TM;
                    held_col = tt * NT;
#pragma unroll
                    for (int i = 0; i < 2; i++) {
#pragma unroll
                        for (int j = 0; j < 4; j++) w[j][i] = w1[j][i];
                        x[i] = x1[i];
                    }
                });
            });
            if (any) write();
        }
    } else {
        // ------------------------------------------------------------------ epilogue
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(RES_EPI_REGS));
        const int qr = warp & 3, cg = (warp >> 2) & 1, h = warp >> 3, col0 = cg * CW;
        const unsigned taddr0 = tmem + ((unsigned)(qr * 32) << 16) + (unsigned)(col0 + 2 * h * SLOT_COLS);
        const unsigned tfull = bars + P_TFULL + 16 * h, tempty = bars + P_TEMPTY + 16 * h;
        float* top = (float*)(base + M::TOP) + tid;     // the last waiting subtree: written and read once a tile
        unsigned slot = 0, phase = 0;
        bool next = false;
        int v[8], sc[8];
        tiles([&](int rt, int tt) {
            f32x2 leaf[2][CW / 2], st[2][CW / 2], x[CW / 2];
            auto visit = [&](int j, f32x2 (&out)[CW / 2]) {   // the rounds of a lane and the lane 16 further, and level s = 16
#pragma unroll
                for (int c = 0; c < CW / 2; c++) leaf[0][c] = leaf[1][c] = 0ull;
#pragma unroll 1
                for (int b = pair_lane(j); b < nb; b += 32) {
                    const unsigned a0 = taddr0 + slot * SLOT_COLS;
                    const unsigned empty = tempty + 8 * slot;
                    bar_wait(next, tfull + 8 * slot, phase, abort_flag, P.status);
                    tc_fence_after();
                    slot ^= 1;
                    if (slot == 0) phase ^= 1;
#pragma unroll
                    for (int i = 0; i < 4; i++) {   // block i / 2, 8 columns; the columns this set finishes first
                        const unsigned a = a0 + (i >> 1) * NT + ((i & 1) ^ h) * 8;
                        tmem_ld_pair(a, a + 2 * NT, v, sc);
                        if (i == 1) next = bar_test(tfull + 8 * slot, phase);
                        if (i == 3) {
                            tc_fence_before();
                            __syncwarp();
                            bar_arrive_if(lane == 0, empty);
                        }
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            f32x2& acc = leaf[i >> 1][(i & 1) * 4 + c];
                            const f32x2 f = pack2((float)v[2 * c], (float)v[2 * c + 1]);
                            acc = fma2(pack2(__int_as_float(sc[2 * c]), __int_as_float(sc[2 * c + 1])), f, acc);
                        }
                    }
                }
#pragma unroll
                for (int c = 0; c < CW / 2; c++) out[c] = add2(leaf[0][c], leaf[1][c]);
            };
            auto join = [&](f32x2 (&left)[CW / 2], f32x2 (&right)[CW / 2], f32x2 (&out)[CW / 2]) {
#pragma unroll
                for (int c = 0; c < CW / 2; c++) out[c] = add2(left[c], right[c]);
            };
            float y[CW];
#pragma unroll 1
            for (int g = 0; g < 2; g++) {
                visit(4 * g, st[0]);
                visit(4 * g + 1, x);
                join(st[0], x, st[1]);
                visit(4 * g + 2, st[0]);
                visit(4 * g + 3, x);
                join(st[0], x, x);
                join(st[1], x, x);
                if (g == 0) {
#pragma unroll
                    for (int c = 0; c < CW / 2; c++) {
                        unpack2(x[c], y[2 * c], y[2 * c + 1]);
                        top[(2 * c) * 512] = y[2 * c];
                        top[(2 * c + 1) * 512] = y[2 * c + 1];
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < CW / 2; c++) x[c] = add2(pack2(top[(2 * c) * 512], top[(2 * c + 1) * 512]), x[c]);
            // the level of the two sets: this one finishes the columns 8 h .. 8 h + 7 of each group of 16, its first four pairs
#pragma unroll
            for (int c = 0; c < CW / 2; c++) unpack2(x[c], y[2 * c], y[2 * c + 1]);
            const int r = qr * 32 + lane, row = rt * TM + r;
            float* xp = xchg + (cg * 16) * TM + r;      // [group][set that finishes][8][row]
            asm volatile("bar.sync 1, %0;" ::"n"(2 * EW * 32) : "memory");   // the last tile's partials have been read
#pragma unroll
            for (int c = 0; c < 8; c++) xp[((1 - h) * 8 + c) * TM] = y[8 + c];
            asm volatile("bar.sync 2, %0;" ::"n"(2 * EW * 32) : "memory");
            const int first = tt * NT + col0 + 8 * h;
            float z[8];
#pragma unroll
            for (int c = 0; c < 8; c++) z[c] = __fadd_rn(y[c], xp[(h * 8 + c) * TM]);
            const int valid = P.T - first;
            if (valid > 0) repair<8>(P, row, first, valid, z);
            if (row < P.M && valid > 0) {
                if (P.Resid != nullptr) {
                    const float* rp = P.Resid + (long)first * P.resid_ld + row;
#pragma unroll
                    for (int c = 0; c < 8; c++, rp += P.resid_ld)
                        if (c < valid) z[c] = __fadd_rn(z[c], *rp);
                }
                float* yp = P.Y + (long)first * P.M + row;
#pragma unroll
                for (int c = 0; c < 8; c++, yp += P.M)
                    if (c < valid) *yp = z[c];
            }
        });
    }

    // ---------------------------------------------------------------------- teardown
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && warp == 2 * EW + 1 && lane == 0) {   // bulk copies still in flight land before the CTA leaves
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) {
        }
    }
    __syncthreads();
    if (warp == 2 * EW) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((unsigned)(NSLOT * SLOT_COLS))
                     : "memory");
    }
}

// ---------------------------------------------------------------------------- host side

static int fill(Params& P, CUtensorMap& tmW, CUtensorMap& tmX, const Args& a, int box_w, int box_x) {
    int rc = make_map(&tmW, a.Wq, a.M, a.K, box_w, TM);
    if (rc != LT_OK) return rc;
    rc = make_map(&tmX, a.Xq, a.T, a.K, box_x, NT);
    if (rc != LT_OK) return rc;
    P.Wd = a.Wd; P.Xd = a.Xd; P.Wq = a.Wq; P.Xq = a.Xq; P.Resid = a.Resid; P.Y = a.Y;
    P.status = device_status_ptr();
    LT_REQUIRE(P.status != nullptr, "lt_q8_gemm_tc: status word unavailable");
    P.M = a.M; P.K = a.K; P.T = a.T; P.resid_ld = a.resid_ld;
    P.col_tiles = (a.T + NT - 1) / NT;
    P.units = (a.M + TM - 1) / TM * P.col_tiles;
    return LT_OK;
}

static bool resident(int K) { return K >= 512 && K <= RES_MAX_K; }   // an l without any block would leave its stage unwritten

bool fits(int M, int K, int T) {
    const long units = (long)((M + TM - 1) / TM) * ((T + NT - 1) / NT);
    return units < (1L << 31) && (long)M * (K / 32) < (1L << 32) && (long)T * (K / 32) < (1L << 32);
}

// Microseconds of a call: launch, and per round of CTAs a tile's end and its steps (of 292 shapes from 128 x 512 to 128256 x 4096
// and 9 to 2048 columns 95 % are within 11 %, all within 15 %).
double cost(int M, int K, int T, int sms) {
    const long units = (long)((M + TM - 1) / TM) * ((T + NT - 1) / NT), rounds = (units + sms - 1) / sms;
    if (resident(K)) return 4.8 + (double)rounds * (0.1 + 0.54 * 8);
    long steps = 0;
    for (int l = 0; l < 16; l += 2) steps += K / 32 > l ? (K / 32 - l + 31) / 32 : 0;
    return 4.5 + (double)rounds * (1.5 + 0.47 * (double)steps);
}

int run(const Args& a, cudaStream_t s) {
    CUtensorMap tmW, tmX;
    Params P;
    LT_REQUIRE(fits(a.M, a.K, a.T), "lt_q8_gemm_tc: M=%d K=%d T=%d have too many tiles", a.M, a.K, a.T);
    const bool res = resident(a.K);
    const int rc = res ? fill(P, tmW, tmX, a, 32, 128) : fill(P, tmW, tmX, a, 64, 64);
    if (rc != LT_OK) return rc;
    static PerDeviceOnce attr_once;
    if (attr_once.first()) {
        LT_CUDA(cudaFuncSetAttribute(k_q8_gemm_res, cudaFuncAttributeMaxDynamicSharedMemorySize, ResSmem(RES_MAX_K / 32).total + 1024));
        LT_CUDA(cudaFuncSetAttribute(k_q8_gemm_pair, cudaFuncAttributeMaxDynamicSharedMemorySize, PairSmem::TOTAL + 1024));
    }
    const int sms = sm_count(), grid = P.units < sms ? P.units : sms;
    if (res) k_q8_gemm_res<<<grid, RES_THREADS, ResSmem(a.K / 32).total + 1024, s>>>(tmW, tmX, P);
    else k_q8_gemm_pair<<<grid, P_THREADS, PairSmem::TOTAL + 1024, s>>>(tmW, tmX, P);
    return check_launch("lt_q8_gemm_tc");
}

}  // namespace pair
}  // namespace tc
}  // namespace lt
