// Q8_0 skinny GEMM / prefill GEMM on the 5th-generation tensor cores (tcgen05, kind::i8).
//
// Same arithmetic contract as the GEMV (lt_gemv.cu), per output row n and activation column t:
//   lane L in 0..31:  acc_L = 0;  for b = L, L+32, ... < K/32 (ascending):
//       isum  = sum_i Wq[n, 32b+i] * Xq[t, 32b+i]                    (exact int32)
//       acc_L = fma( f32(Wd[n,b]) * f32(Xd[t,b]), (float)isum, acc_L )
//   Y[t, n] = tree over the 32 lane values, s = 16, 8, 4, 2, 1: acc_l += acc_{l+s}   (+ Resid[n])
//
// The integer part is the dense contraction: one tcgen05.mma (M = 128 weight rows, N = NT
// activation columns, K = 32 bytes) produces the isum of one Q8_0 block for 128 x NT outputs as
// int32 in tensor memory.  Each block needs its own accumulator (the fp32 scale differs per
// block), so the fp32 part runs on the CUDA cores: epilogue warps read a block's 128 x NT int32
// from TMEM, scale and fold them in exactly the order above.  The "lanes" of the contract are
// plain registers here: thread = one weight row (TMEM lane) x CW columns, and the blocks are
// visited so that a row needs few live partials:
//   groups of CB adjacent lanes (CB blocks = one shared-memory chunk of CB*32 bytes per row) are
//   visited in bit-reversed group order; inside a group the rounds r = 0, 1, ... (block
//   CB*g + i + 32 r) extend the CB lane accumulators in ascending order; a finished group is
//   pushed on a log2(32/CB)-deep stack that performs the s = 16, 8, ... levels of the tree as
//   soon as both operands exist; the last log2(CB) levels combine the CB stacks at the end.
//
// Pipeline per CTA (persistent over tiles of 128 rows x NT columns):
//   warp EW   : producer, TMA tiled loads (hardware swizzle) of weight and activation chunks
//               into a ring of shared-memory stages; a stage = one chunk of CB blocks
//   warp EW+1 : one thread issues the CB MMAs of a stage into a ring of TMEM slots and commits
//   warps 0..EW-1 : epilogue, TMEM -> registers -> fp32 fold -> Y
// Split rows of blocks (S > 1): a cluster of S CTAs shares a tile, CTA r visits the groups g = r mod S, a whole subtree of
// the tree; the levels across those subtrees and inside a group are added by the CTA that finishes a column, from all
// CTAs' partials in its shared memory.  Small batches need it: a matrix of 4096 rows has 32 row tiles for 148 SMs
// (4096 x 14336, 24 columns: 64 CTAs 55 us, 128 CTAs 34 us; 9 columns: 32 CTAs 66 us, 128 CTAs 28 us).
// Every wait is bounded: after the limit a CTA sets LT_STATUS_WAIT_TIMEOUT, all its later waits
// return at once, it drains and frees its tensor memory.
#include <atomic>

#include "lt_gemm_pair.cuh"
#include "lt_tc.cuh"

namespace lt {
namespace tc {

constexpr int TM = 128;          // weight rows per tile (MMA M, TMEM lanes)
constexpr int TMEM_COLS = 256;   // allocated tensor-memory columns (two CTAs may share an SM)

// the wait after the loads of CB blocks of CW columns, every register passed through it
template <int N, int CB, int CW>
__device__ __forceinline__ void tmem_ld_wait(int (&v)[CB][CW]) {
    static_assert(N == CB * CW && CW % 4 == 0, "register count");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < CB; i++)
#pragma unroll
        for (int c = 0; c < CW; c += 4) reg_fence4(&v[i][c]);
}

// ---- cluster
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned map_rank(unsigned addr, unsigned rank) {   // the same shared address in another CTA of the cluster
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void arrive_remote(unsigned bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool try_wait_cluster(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void wait_cluster(unsigned long long* bar, unsigned parity, volatile int* abort_flag, int* status) {
    if (try_wait_cluster(bar, parity)) return;
    const long long t0 = clock64();
    while (!try_wait_cluster(bar, parity)) {
        if (*abort_flag) return;
        if (clock64() - t0 > WAIT_LIMIT) {
            *abort_flag = 1;
            atomicOr(status, LT_STATUS_WAIT_TIMEOUT);
            return;
        }
    }
}

constexpr int ilog2(int v) { return v <= 1 ? 0 : 1 + ilog2(v >> 1); }

struct Params {
    const __half* Wd;
    const __half* Xd;
    const float* Resid;
    float* Y;
    int* status;
    int M, K, T;
    int row_tiles, t_tiles;
    int resid_ld;   // 0: Resid[n] for every column (bias); else Resid[t * resid_ld + n]
};

template <int NT, int CB, int EW, int S, int NST>      // NST: stages of the ring
struct Cfg {
    static constexpr int CW = NT * 4 / EW;             // columns per epilogue thread
    static constexpr int G = 32 / CB / S;              // lane groups that a CTA of the cluster visits
    static constexpr int LV = ilog2(G);                // stack depth
    static constexpr int QPR = NT / 4 / S;             // quads of columns that a CTA finishes
    static constexpr int XCHG = S > 1 ? S * QPR * CB * TM * 16 : 0;   // bytes of the partials of those columns
    static constexpr int MW = 2;                       // MMA-issuing warps
    static constexpr int THREADS = (EW + 1 + MW) * 32;
    static constexpr int W_STAGE = CB * TM * 32;       // bytes: one stage = one chunk of CB blocks
    static constexpr int X_STAGE = CB * NT * 32;
    static constexpr int STAGE = W_STAGE + ((X_STAGE + 1023) / 1024) * 1024;
    static constexpr int SLOT_COLS = CB * NT;
    static constexpr int NSLOT = TMEM_COLS / SLOT_COLS;
    static constexpr int LB = CB * CW <= 16 ? CB : (CB >= 2 && CW <= 8 ? 2 : 1);   // blocks per TMEM round trip
    static_assert(EW % 4 == 0 && (CW == 4 || CW == 8 || CW == 16), "epilogue shape");
    static_assert(NSLOT >= 2 && NSLOT <= 16 && (NSLOT & (NSLOT - 1)) == 0, "TMEM slots");
    static_assert(W_STAGE % 1024 == 0, "stages keep 1024-byte alignment");
    static_assert(S == 1 || (EW == 8 && CW == 8 && NT == 16 && (S == 2 || S == 4)), "the exchange deals quads to ranks");
};

struct Barriers {
    unsigned long long full[8], empty[8];
    unsigned long long tfull[16], tempty[16];
    unsigned tmem_base;
    int abort_flag;
    unsigned long long xfull, xfree[4];   // all partials of this CTA's columns are here; rank r has read what it was sent
    int next_start[32];   // per visiting position: first block of the next group that has blocks, -1 = none
};

template <int NT, int CB, int EW, int S, int NSTAGE>
__global__ void __launch_bounds__(Cfg<NT, CB, EW, S, NSTAGE>::THREADS, 1)
k_q8_gemm_tc(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const Params P) {
    using C = Cfg<NT, CB, EW, S, NSTAGE>;
    constexpr int CW = C::CW, G = C::G, LV = C::LV, NSLOT = C::NSLOT, LB = C::LB, MW = C::MW;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // 1024-byte aligned carve-up: stages (weights, then activations), barriers, exchange, activation scales
    unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    Barriers* B = (Barriers*)(base + NSTAGE * C::STAGE);
    float* xchg = (float*)((unsigned char*)B + 1024);
    float* xs = (float*)((unsigned char*)xchg + C::XCHG);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nb = P.K >> 5;
    const int tiles = P.row_tiles * P.t_tiles;
    const int rank = S > 1 ? (int)cluster_rank() : 0;
    const int tile_first = blockIdx.x / S, tile_step = gridDim.x / S;
    auto group = [&](int gi) {   // the gi-th group this CTA visits
        return rank + S * (LV > 0 ? (int)(__brev((unsigned)gi) >> (32 - (LV > 0 ? LV : 1))) : 0);
    };
    // of a tile, in this CTA: every S-th chunk
    const unsigned chunks = (unsigned)((nb / CB + S - 1 - rank) / S);
    volatile int* abort_flag = &B->abort_flag;

    if (warp == 0) {   // a lane per barrier and per visiting position: one thread alone takes 0.2 us longer
        if (lane < NSTAGE) {
            mbar_init(&B->full[lane], 1);
            mbar_init(&B->empty[lane], 1);
        }
        if (lane < NSLOT) {
            mbar_init(&B->tfull[lane], 1);
            mbar_init(&B->tempty[lane], EW);
        }
        if (S > 1 && lane < S) mbar_init(&B->xfree[lane], EW);
        if (lane == 0) {
            if (S > 1) mbar_init(&B->xfull, 4 * S);
            B->abort_flag = 0;
        }
        if (lane < G) {
            int nxt = -1;
            for (int gj = G - 1; gj > lane; gj--) {
                const int b0 = CB * group(gj);
                if (b0 < nb) nxt = b0;
            }
            B->next_start[lane] = nxt;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == EW + 1) {   // the MMA warp owns the tensor-memory allocation
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&B->tmem_base)),
                     "r"((unsigned)TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncwarp();
    if (S > 1) cluster_sync();   // the other CTAs' barriers are initialised
    else __syncthreads();
    tc_fence_after();
    const unsigned tmem = B->tmem_base;

    // chunks per tile: groups in bit-reversed order, rounds ascending; identical in all three roles
    if (warp == EW) {
        // ------------------------------------------------------------------ producer
        if (lane == 0) {
            unsigned it = 0;   // chunks issued
            for (int tile = tile_first; tile < tiles; tile += tile_step) {
                const int rt = tile / P.t_tiles, tt = tile - rt * P.t_tiles;
                const int row0 = rt * TM, t0 = tt * NT;
                for (int gi = 0; gi < G; gi++) {
                    const int g = group(gi);
                    for (int b0 = CB * g; b0 < nb; b0 += 32, it++) {
                        const int s = it % NSTAGE;
                        unsigned char* st = base + s * C::STAGE;
                        mbar_wait<64>(&B->empty[s], ((it / NSTAGE) & 1) ^ 1, abort_flag, P.status);
                        mbar_expect_tx(&B->full[s], C::W_STAGE + C::X_STAGE);
                        tma_load_2d(st, &tmW, b0 * 32, row0, &B->full[s]);
                        tma_load_2d(st + C::W_STAGE, &tmX, b0 * 32, t0, &B->full[s]);
                    }
                }
            }
        }
    } else if (warp >= EW + 1) {
        // ------------------------------------------------------------------ MMA issue
        // MW warps share the chunks round-robin (a chunk has its own stage and slot, so the warps
        // are independent); issuing, not the tensor pipe, limits these small MMAs.
        if (lane == 0) {
            // instruction descriptor: D = s32, A = B = signed 8-bit, both K-major, N = NT, M = 128
            constexpr unsigned idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(NT >> 3) << 17) |
                                       ((unsigned)(TM >> 4) << 24);
            const unsigned long long wdesc0 = smem_desc<CB>(smem_u32(base));
            const unsigned long long xdesc0 = smem_desc<CB>(smem_u32(base) + C::W_STAGE);
            int my_tiles = 0;
            for (int tile = tile_first; tile < tiles; tile += tile_step) my_tiles++;
            const unsigned total = (unsigned)my_tiles * chunks;
            for (unsigned it = (unsigned)(warp - (EW + 1)); it < total; it += MW) {
                const unsigned s = it % NSTAGE, slot = it % NSLOT;
                mbar_wait<32>(&B->full[s], (it / NSTAGE) & 1, abort_flag, P.status);
                mbar_wait<32>(&B->tempty[slot], ((it / NSLOT) & 1) ^ 1, abort_flag, P.status);
                tc_fence_after();
                // descriptors differ from the first stage's only in the start address (16-byte units)
                const unsigned long long wd0 = wdesc0 + (unsigned long long)(s * (C::STAGE >> 4));
                const unsigned long long xd0 = xdesc0 + (unsigned long long)(s * (C::STAGE >> 4));
                const unsigned d0 = tmem + slot * C::SLOT_COLS;
#pragma unroll
                for (int i = 0; i < CB; i++)   // block i = the i-th 32-byte slice of the swizzled rows
                    mma_i8(d0 + i * NT, wd0 + 2 * i, xd0 + 2 * i, idesc);
                mma_commit(&B->empty[s]);     // the stage may be refilled once these MMAs have read it
                mma_commit(&B->tfull[slot]);  // and the slot holds the block sums
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue
        // A thread walks its row's blocks in the visiting order.  While it folds a block, the
        // TMEM load of the next block and the global load of the next weight scales are in flight.
        const int q = warp & 3, cg = warp >> 2;
        const int col0 = cg * CW;
        const unsigned lane_addr = ((unsigned)(q * 32) << 16) + (unsigned)col0;
        int my_tiles = 0;
        for (int tile = tile_first; tile < tiles; tile += tile_step) my_tiles++;
        const unsigned total = (unsigned)my_tiles * chunks;                // chunks this thread consumes
        unsigned it = 0;                                                   // chunks consumed so far
        unsigned turn = 0;                                                 // tiles exchanged so far
        auto scale_row = [&](int tile) {   // this thread's row of weight scales in a tile (row 0 if out of range)
            int r = (tile / P.t_tiles) * TM + q * 32 + lane;
            if (r >= P.M) r = 0;
            return P.Wd + (long)r * nb;
        };
        auto scales_at = [&](const __half* p) {   // the CB scales of blocks b .. b+CB-1
            uint2 w = make_uint2(0u, 0u);
            if (CB == 4) w = __ldg((const uint2*)p);
            else if (CB == 2) w.x = __ldg((const unsigned*)p);
            else w.x = __ldg((const unsigned short*)p);
            return w;
        };
        uint2 wnext = make_uint2(0u, 0u);
        if (total > 0) wnext = scales_at(scale_row(tile_first) + CB * rank);

        for (int tile = tile_first; tile < tiles; tile += tile_step) {
            const int rt = tile / P.t_tiles, tt = tile - rt * P.t_tiles;
            const int row = rt * TM + q * 32 + lane, t0 = tt * NT;
            const bool row_ok = row < P.M;
            const __half* wdrow = scale_row(tile);
            const __half* wdrow_next = scale_row(tile + tile_step < tiles ? tile + tile_step : tile) + CB * rank;

            // activation scales of this column tile: xs[b][c] = f32(Xd[t0 + c, b])
            asm volatile("bar.sync 1, %0;" ::"n"(EW * 32) : "memory");
            for (int c = warp; c < NT; c += EW) {
                const bool ok = t0 + c < P.T;
                const __half* xr = P.Xd + (long)(ok ? t0 + c : 0) * nb;
                for (int b = lane; b < nb; b += 32)
                    if (S == 1 || ((b / CB) & (S - 1)) == rank) xs[b * NT + c] = ok ? __half2float(xr[b]) : 0.0f;
            }
            asm volatile("bar.sync 1, %0;" ::"n"(EW * 32) : "memory");

            float stack[CB][LV > 0 ? LV : 1][CW];
            float fin[CB][CW];
#pragma unroll
            for (int gi = 0; gi < G; gi++) {
                const int g = group(gi);
                float leaf[CB][CW];
#pragma unroll
                for (int i = 0; i < CB; i++)
#pragma unroll
                    for (int c = 0; c < CW; c++) leaf[i][c] = 0.0f;

                for (int b0 = CB * g; b0 < nb; b0 += 32) {
                    const uint2 wcur = wnext;
                    {   // scales of the next chunk: next round of this group, else the next group that
                        // has blocks, else the first chunk of the next tile
                        const __half* np = wdrow + b0 + 32;
                        if (b0 + 32 >= nb) {
                            const int ns = B->next_start[gi];
                            np = ns < 0 ? wdrow_next : wdrow + ns;
                        }
                        wnext = scales_at(np);
                    }
                    // all CB blocks of the chunk in one round trip to tensor memory
                    const unsigned slot = it % NSLOT;
                    const unsigned taddr = tmem + lane_addr + slot * C::SLOT_COLS;
                    mbar_wait(&B->tfull[slot], (it / NSLOT) & 1, abort_flag, P.status);
                    tc_fence_after();
#pragma unroll
                    for (int h = 0; h < CB; h += LB) {   // LB blocks per round trip to tensor memory
                        int v[LB][CW];
#pragma unroll
                        for (int i = 0; i < LB; i++) tmem_ld<CW>(taddr + (h + i) * NT, v[i]);
                        tmem_ld_wait<LB * CW>(v);
                        if (h + LB == CB) {
                            // the chunk's sums are in registers: hand the slot back to the MMA warp
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&B->tempty[slot]);
                            it++;
                        }
#pragma unroll
                        for (int j = 0; j < LB; j++) {
                            const int i = h + j;
                            const unsigned short wbits =
                                CB == 4 ? (unsigned short)((i < 2 ? wcur.x : wcur.y) >> ((i & 1) * 16))
                                        : (unsigned short)(wcur.x >> ((i & 1) * 16));
                            const float wd = __half2float(__ushort_as_half(wbits));
                            const float4* xp = (const float4*)(xs + (b0 + i) * NT + col0);
#pragma unroll
                            for (int c4 = 0; c4 < CW / 4; c4++) {
                                const float4 x = xp[c4];
                                leaf[i][4 * c4] = __fmaf_rn(__fmul_rn(wd, x.x), (float)v[j][4 * c4], leaf[i][4 * c4]);
                                leaf[i][4 * c4 + 1] =
                                    __fmaf_rn(__fmul_rn(wd, x.y), (float)v[j][4 * c4 + 1], leaf[i][4 * c4 + 1]);
                                leaf[i][4 * c4 + 2] =
                                    __fmaf_rn(__fmul_rn(wd, x.z), (float)v[j][4 * c4 + 2], leaf[i][4 * c4 + 2]);
                                leaf[i][4 * c4 + 3] =
                                    __fmaf_rn(__fmul_rn(wd, x.w), (float)v[j][4 * c4 + 3], leaf[i][4 * c4 + 3]);
                            }
                        }
                    }
                }
                // push the finished group: levels whose left operand is already there are added now
#pragma unroll
                for (int i = 0; i < CB; i++) {
                    bool placed = false;
#pragma unroll
                    for (int lv = 0; lv < LV; lv++) {
                        if (!placed) {
                            if ((gi >> lv) & 1) {
#pragma unroll
                                for (int c = 0; c < CW; c++) leaf[i][c] = __fadd_rn(stack[i][lv][c], leaf[i][c]);
                            } else {
#pragma unroll
                                for (int c = 0; c < CW; c++) stack[i][lv][c] = leaf[i][c];
                                placed = true;
                            }
                        }
                    }
                    if (!placed) {
#pragma unroll
                        for (int c = 0; c < CW; c++) fin[i][c] = leaf[i][c];
                    }
                }
            }
            if (S > 1) {
                // this thread's CB x CW partials go to the CTAs that finish the columns, by quads:
                // [source rank][quad of the rank][lane of the group][row][4]
                constexpr int QPR = C::QPR;
                const int r = q * 32 + lane;
#pragma unroll
                for (int h = 0; h < CW / 4; h++) {
                    const unsigned quad = (unsigned)(cg * (CW / 4) + h), dst = quad / QPR;
                    wait_cluster(&B->xfree[dst], (turn & 1) ^ 1, abort_flag, P.status);
                    const unsigned buf = map_rank(smem_u32(xchg), dst) + ((unsigned)rank * QPR + quad % QPR) * (CB * TM * 16);
#pragma unroll
                    for (int i = 0; i < CB; i++)
                        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(buf + (unsigned)((i * TM + r) * 16)),
                                     "f"(fin[i][4 * h]), "f"(fin[i][4 * h + 1]), "f"(fin[i][4 * h + 2]), "f"(fin[i][4 * h + 3])
                                     : "memory");
                    // one arrival per warp and destination (both quads of a warp may have the same)
                    if (QPR == 1 || h == CW / 4 - 1) {
                        __syncwarp();
                        if (lane == 0) arrive_remote(map_rank(smem_u32(&B->xfull), dst));
                    }
                }
                wait_cluster(&B->xfull, turn & 1, abort_flag, P.status);
                // columns 4 * QPR * rank + cg * NC ..: levels across the ranks, then across the lanes of a group
                constexpr int NC = 2 * QPR;
                float y[NC];
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    const int col = cg * NC + c;      // among this rank's columns
                    float part[CB];
#pragma unroll
                    for (int i = 0; i < CB; i++) {
                        float pr[S];
#pragma unroll
                        for (int k = 0; k < S; k++) pr[k] = xchg[(((k * QPR + col / 4) * CB + i) * TM + r) * 4 + col % 4];
#pragma unroll
                        for (int s = S / 2; s >= 1; s >>= 1)
#pragma unroll
                            for (int k = 0; k < s; k++) pr[k] = __fadd_rn(pr[k], pr[k + s]);
                        part[i] = pr[0];
                    }
#pragma unroll
                    for (int s = CB / 2; s >= 1; s >>= 1)
#pragma unroll
                        for (int i = 0; i < s; i++) part[i] = __fadd_rn(part[i], part[i + s]);
                    y[c] = part[0];
                }
                __syncwarp();
                if (lane < S) arrive_remote(map_rank(smem_u32(&B->xfree[rank]), (unsigned)lane));
                turn++;
                if (row_ok) {
#pragma unroll
                    for (int c = 0; c < NC; c++) {
                        const int t = t0 + 4 * QPR * rank + cg * NC + c;
                        if (t < P.T) {
                            if (P.Resid != nullptr) y[c] = __fadd_rn(y[c], P.Resid[(long)t * P.resid_ld + row]);
                            P.Y[(long)t * P.M + row] = y[c];
                        }
                    }
                }
                continue;
            }
            // last levels of the tree across the CB lanes of a group: strides CB/2, ..., 1
#pragma unroll
            for (int s = CB / 2; s >= 1; s >>= 1)
#pragma unroll
                for (int i = 0; i < s; i++)
#pragma unroll
                    for (int c = 0; c < CW; c++) fin[i][c] = __fadd_rn(fin[i][c], fin[i + s][c]);

            if (row_ok) {
#pragma unroll
                for (int c = 0; c < CW; c++) {
                    const int t = t0 + col0 + c;
                    if (t < P.T) {
                        float y = fin[0][c];
                        if (P.Resid != nullptr) y = __fadd_rn(y, P.Resid[(long)t * P.resid_ld + row]);
                        P.Y[(long)t * P.M + row] = y;
                    }
                }
            }
        }
    }

    // ---------------------------------------------------------------------- teardown
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && warp == EW && lane == 0) {
        // a wait ran out: give bulk copies still in flight time to land before the CTA leaves
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) {
        }
    }
    __syncwarp();
    if (S > 1) cluster_sync();   // no CTA leaves while another may still write to its shared memory
    else __syncthreads();
    if (warp == EW + 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((unsigned)TMEM_COLS)
                     : "memory");
    }
}

// ---------------------------------------------------------------------------- host side

int make_map(CUtensorMap* m, const void* ptr, int rows, int K, int box_k, int box_rows) {
    encode_fn_t fn = encode_fn();
    if (fn == nullptr) {
        set_error("lt_q8_gemm_tc: cuTensorMapEncodeTiled is not available from this driver");
        return LT_ERR_CUDA;
    }
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)K};
    cuuint32_t box[2] = {(cuuint32_t)box_k, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUtensorMapSwizzle sw = box_k == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                                         : (box_k == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("lt_q8_gemm_tc: cuTensorMapEncodeTiled failed (%d) for rows=%d K=%d box=%dx%d", (int)r, rows, K,
                  box_k, box_rows);
        return LT_ERR_CUDA;
    }
    return LT_OK;
}

// ---- how many CTAs share a 16-column tile
// A tile of c chunks costs a round of CTAs, in microseconds (28 shapes from 128 x 512 to 16384 x 7168, 9 to 1500 columns):
// alone 0.455 c + 1; two CTAs 0.5 c / 2 + 3; four 0.55 c / 4 + 4 (the exchange, and pairs that share what the L2 delivers).
// 4096 x 14336: 9 columns 66 us alone, 37 with two, 28 with four; 24 columns 55, 34, 47; 33 columns 53, 65, 68; 96 columns
// 108, 92, 134; 896 x 896: 6.3, 6.8, 7.3.  Four CTAs pay only in a single round, as measured: with more, two are better.
// rooms[]: clusters of 2 and 4 that the GPU holds at once.  Four need SMs of one GPC, and the last few of the GPC counts that
// are no multiple of four stay alone: 33 clusters on 148 SMs.  A launch takes no more clusters than that, since tiles are
// dealt out in advance and the clusters that wait for a place would start when the others end.
static double split_cost(int S, long tiles, int chunks, long room) {
    if (room < 1) return 1e30;
    const long rounds = (tiles + room - 1) / room;
    if (S == 4 && rounds > 1) return 1e30;
    const double c = (double)((chunks + S - 1) / S);
    return (double)rounds * (S == 1 ? 0.455 * c + 1.0 : (S == 2 ? 0.5 * c + 3.0 : 0.55 * c + 4.0));
}
// bytes of shared memory of a launch; a CTA may have MAX_SMEM
constexpr size_t MAX_SMEM = 220 * 1024;
template <int NT, int CB, int EW, int S, int NST>
static size_t smem_bytes(int nb) {
    using C = Cfg<NT, CB, EW, S, NST>;
    return 1024 + (size_t)NST * C::STAGE + 1024 + C::XCHG + (size_t)nb * NT * 4;
}
static int choose_split(int M, int K, int T, int sms, int room2, int room4) {
    const int nb = K / 32, chunks = nb / 4;
    const long tiles = (long)((M + TM - 1) / TM) * ((T + 15) / 16);
    if (smem_bytes<16, 4, 8, 2, 6>(nb) > MAX_SMEM) return 1;     // four need less
    const long rooms[3] = {sms, room2, room4};
    int best = 0;
    for (int i = 1; i < 3; i++)
        if (split_cost(1 << i, tiles, chunks, rooms[i]) < split_cost(1 << best, tiles, chunks, rooms[best])) best = i;
    return 1 << best;
}

// The 32-column tiles of lt_gemm_pair.cu where they are faster by more than their times scatter.  Over 292 shapes (15 matrices
// from 128 x 512 to 128256 x 4096, 9 to 2048 columns) the chosen form takes 0.1 % more than the better one on average, at most 9 %
// (1024 x 640 x 512, which stays here at 10.0 us against 9.2), and never more than 2 % over the form here.  Few columns of a
// small matrix stay here: the other kernels' first tile comes 3 us later (896 x 896 x 64 6.8 us, 9.6; x 2048 30, 22;
// 4096 x 4096 x 64 17.1, 20.7; 28672 x 4096 x 32 61, 43).
static bool choose_pair(int M, int K, int T, int sms, int room2, int room4) {
    const int nb = K / 32, S = choose_split(M, K, T, sms, room2, room4);
    const long rooms = S == 4 ? room4 : (S == 2 ? room2 : sms), tiles = (long)((M + TM - 1) / TM) * ((T + 15) / 16);
    // rows too long for the 16-column tiles' scales are refused as before
    if (!pair::fits(M, K, T) || smem_bytes<16, 4, 8, 1, 4>(nb) > MAX_SMEM) return false;
    return 1.05 * pair::cost(M, K, T, sms) + 1.0 < split_cost(S, tiles, nb / 4, rooms) + 3.0;
}

// Eight stages instead of four where a tile has one CTA, if they fit: where a row is long and its weights serve several column
// tiles, which then come from L2 (28672 x 4096 x 512 727 us with four, 684 with eight; 128256 x 4096 x 32 208, 200; 4096 x 4096
// x 1500 313, 293), and for small matrices (9728 x 896 x 9 6.9, 6.5; x 1500 197, 195).  Four where a matrix streams once (65536 x 2048 x 9
// 36.6, 38.7) or is large with rows so short that the ring runs into the next tile (65536 x 896 x 128 113.6, 116.1).  Shared
// tiles take six (4096 x 14336 x 24: 35.0, 33.8, 34.2 with four, six, eight).
static bool deep_ring(int M, int K, int T) {
    const bool small = (long)M * K <= (T > 16 ? 16L : 10L) << 20;
    return (small || (T > 16 && K >= 2048)) && smem_bytes<16, 4, 8, 1, 8>(K / 32) <= MAX_SMEM;
}

// CTAs (S = 1) or clusters of S CTAs that the current device holds at once, asked for once per device
template <int NT, int CB, int EW, int S, int NST>
static int room() {
    static std::atomic<int> known[64];
    int dev = 0;
    if (S == 1 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return sm_count() / S;
    int n = known[dev].load(std::memory_order_relaxed);
    if (n > 0) return n;
    if (cudaFuncSetAttribute(k_q8_gemm_tc<NT, CB, EW, S, NST>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sm_count() / S * S));
    cfg.blockDim = dim3(Cfg<NT, CB, EW, S, NST>::THREADS);
    cfg.dynamicSmemBytes = MAX_SMEM;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = S;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, k_q8_gemm_tc<NT, CB, EW, S, NST>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    known[dev].store(n, std::memory_order_relaxed);
    return n;
}

template <int NT, int CB, int EW, int S, int NST>
static int launch(const int8_t* Wq, const uint16_t* Wd, const int8_t* Xq, const uint16_t* Xd, const float* Resid,
                  int resid_ld, float* Y, int M, int K, int T, cudaStream_t s) {
    using C = Cfg<NT, CB, EW, S, NST>;
    const int nb = K / 32;
    CUtensorMap tmW, tmX;
    int rc = make_map(&tmW, Wq, M, K, CB * 32, TM);
    if (rc != LT_OK) return rc;
    rc = make_map(&tmX, Xq, T, K, CB * 32, NT);
    if (rc != LT_OK) return rc;
    const size_t smem = smem_bytes<NT, CB, EW, S, NST>(nb);
    LT_REQUIRE(smem <= MAX_SMEM, "lt_q8_gemm_tc: K=%d needs %zu bytes of shared memory per CTA", K, smem);
    static PerDeviceOnce attr_once;
    if (attr_once.first()) {
        LT_CUDA(cudaFuncSetAttribute(k_q8_gemm_tc<NT, CB, EW, S, NST>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM));
    }
    Params P;
    P.Wd = (const __half*)Wd; P.Xd = (const __half*)Xd; P.Resid = Resid; P.Y = Y;
    P.status = device_status_ptr();
    LT_REQUIRE(P.status != nullptr, "lt_q8_gemm_tc: status word unavailable");
    P.M = M; P.K = K; P.T = T; P.resid_ld = resid_ld;
    P.row_tiles = (M + TM - 1) / TM;
    P.t_tiles = (T + NT - 1) / NT;
    const long tiles = (long)P.row_tiles * P.t_tiles;
    const int most = room<NT, CB, EW, S, NST>();
    LT_REQUIRE(most > 0, "lt_q8_gemm_tc: this device has no room for clusters of %d", S);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((tiles < most ? tiles : most) * S));
    cfg.blockDim = dim3(C::THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    if (S > 1) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = S;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
    }
    return check_launch("lt_q8_gemm_tc", 1, cudaLaunchKernelEx(&cfg, k_q8_gemm_tc<NT, CB, EW, S, NST>, tmW, tmX, P));
}

}  // namespace tc
}  // namespace lt

using namespace lt;

extern "C" int lt_q8_gemm_tc(const int8_t* Wq, const uint16_t* Wd, const int8_t* Xq, const uint16_t* Xd,
                             const float* Resid, int resid_ld, float* Y, int M, int K, int T, int variant,
                             void* stream) {
    LT_REQUIRE(Wq && Wd && Xq && Xd && Y, "lt_q8_gemm_tc: null pointer");
    LT_REQUIRE(M > 0 && T > 0, "lt_q8_gemm_tc: M=%d T=%d must be positive", M, T);
    LT_REQUIRE(K > 0 && K % 128 == 0, "lt_q8_gemm_tc: K=%d must be a positive multiple of 128", K);
    LT_REQUIRE(aligned16(Wq) && aligned16(Xq), "lt_q8_gemm_tc: Wq and Xq must be 16-byte aligned");
    LT_REQUIRE(resid_ld == 0 || resid_ld >= M, "lt_q8_gemm_tc: resid_ld=%d must be 0 or at least M=%d", resid_ld, M);
    LT_REQUIRE(Resid == nullptr || resid_ld != 0 || T == 1 || (const void*)Y != (const void*)Resid,
               "lt_q8_gemm_tc: Y may alias Resid only when Resid has one row per column");
    cudaStream_t s = (cudaStream_t)stream;
    if (variant == 0) {
        const int room2 = tc::room<16, 4, 8, 2, 6>(), room4 = tc::room<16, 4, 8, 4, 6>();
        const int S = tc::choose_split(M, K, T, sm_count(), room2, room4);
        variant = tc::choose_pair(M, K, T, sm_count(), room2, room4) ? 6 : (S == 4 ? 5 : (S == 2 ? 4 : 1));
    }
    if (variant == 1 && tc::deep_ring(M, K, T)) return tc::launch<16, 4, 8, 1, 8>(Wq, Wd, Xq, Xd, Resid, resid_ld, Y, M, K, T, s);
    if (variant == 1) return tc::launch<16, 4, 8, 1, 4>(Wq, Wd, Xq, Xd, Resid, resid_ld, Y, M, K, T, s);
    if (variant == 2) return tc::launch<32, 1, 8, 1, 8>(Wq, Wd, Xq, Xd, Resid, resid_ld, Y, M, K, T, s);
    if (variant == 3) return tc::launch<16, 4, 16, 1, 4>(Wq, Wd, Xq, Xd, Resid, resid_ld, Y, M, K, T, s);
    if (variant == 4) return tc::launch<16, 4, 8, 2, 6>(Wq, Wd, Xq, Xd, Resid, resid_ld, Y, M, K, T, s);
    if (variant == 5) return tc::launch<16, 4, 8, 4, 6>(Wq, Wd, Xq, Xd, Resid, resid_ld, Y, M, K, T, s);
    if (variant == 6) return tc::pair::run({Wq, Xq, Wd, Xd, Resid, resid_ld, Y, M, K, T}, s);
    set_error("lt_q8_gemm_tc: unknown variant %d", variant);
    return LT_ERR_INVALID;
}

extern "C" int lt_q8_gemm_tc_pair(int M, int K, int T, int sms, int clusters2, int clusters4) {
    return M > 0 && K > 0 && K % 128 == 0 && T > 0 && sms > 0 && tc::choose_pair(M, K, T, sms, clusters2, clusters4);
}

extern "C" int lt_q8_gemm_tc_split(int M, int K, int T, int sms, int clusters2, int clusters4) {
    return M > 0 && K > 0 && K % 128 == 0 && T > 0 && sms > 0 ? tc::choose_split(M, K, T, sms, clusters2, clusters4) : 0;
}

