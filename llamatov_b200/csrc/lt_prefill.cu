// Row-batched forms of the decode operators, for prefilling a prompt in one pass.
//
// The reference prefills by running its one-token step once per prompt token
// (bpd/lib/dev_residency.py:1344-1350) and requires any batched form to give the same
// numbers.  Every kernel here therefore computes, for row r of the batch, exactly what the
// one-token kernel computes for that token: same fold orders, same device functions.  What
// changes is only how the work is spread: rows share one launch, and the causal attention
// reads each cached K/V row once per tile of query rows instead of once per query.
#include "lt_common.cuh"
#include "lt_device_ops.cuh"

namespace lt {

// ------------------------------------------------------------------ embedding rows
__global__ void k_embed_q8_rows(const int8_t* __restrict__ Wq, const __half* __restrict__ Wd,
                                const int* __restrict__ toks, float* __restrict__ out, int E, int V, int nrows,
                                int* status) {
    chain_release();
    chain_wait();
    const int r = blockIdx.x;
    if (r >= nrows) return;
    int t = toks[r];
    if (t < 0 || t >= V) {
        if (threadIdx.x == 0) atomicOr(status, (int)LT_STATUS_BAD_TOKEN);
        t = t < 0 ? 0 : V - 1;
    }
    const int nb = E >> 5;
    for (int i = threadIdx.x; i < E; i += blockDim.x) {
        const float q = (float)Wq[(long)t * E + i];
        const float d = __half2float(Wd[(long)t * nb + (i >> 5)]);
        out[(long)r * E + i] = __fmul_rn(q, d);
    }
}

// ------------------------------------------------------------------ rope rows
// row r of X (row stride ld floats, n_head heads of hd at the row start) is rotated at position *pos0 + r
__global__ void k_rope_rows(float* __restrict__ X, int ld, const int* __restrict__ pos0, int nrows, int n_head, int hd,
                            float theta) {
    const int half = hd / 2;
    const long total = (long)nrows * n_head * half;
    const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= total) return;
    const int j = gid % half;
    const long hr = gid / half;
    const int head = hr % n_head;
    const int row = hr / n_head;
    const long base = (long)row * ld + (long)head * hd;
    float o1, o2;
    rope_pair(X[base + j], X[base + j + half], j, hd, theta, *pos0 + row, o1, o2);
    X[base + j] = o1;
    X[base + j + half] = o2;
}

// ------------------------------------------------------------------ rope + KV append of several sequences
// Rows b * T + r of X (q heads, k heads, v heads of hd) are rotated at position start[b] + r, k and v go to the caches' rows from
// start[b] on, the lengths become start[b] + T.  A thread has one pair of every head of its part of a row, so that the angle
// (a power, a sine and a cosine: what k_rope_rows spends its time on) is worked out once for all of them.  2048 rows of 14 + 2 + 2
// heads of 64: 16.4 us in three launches (rotation 11.7), 6.6 here; three sequences of 333 rows 21.5 us in nine, 5.0 here.
__global__ void __launch_bounds__(256) k_rope_append_rows(float* __restrict__ X, int ld, const __grid_constant__ lt_row_seqs S, int B,
                                                          int T, int nh, int nkv, int hd, float theta, int per) {
    const int half = hd / 2, width = nkv * hd;
    const long gid = (long)blockIdx.x * 256 + threadIdx.x;
    const int row = (int)(gid / half), j = (int)(gid - (long)row * half);
    if (row >= B * T) return;
    const int b = row / T, r = row - b * T, pos = S.start[b] + r;
    if (r == 0 && j == 0 && blockIdx.y == 0) *S.len[b] = S.start[b] + T;
    float c, s;
    rope_trig(j, hd, theta, pos, c, s);
    const int h1 = min((int)(blockIdx.y + 1) * per, nh + 2 * nkv);
#pragma unroll 4
    for (int h = blockIdx.y * per; h < h1; h++) {
        float* x = X + (long)row * ld + (long)h * hd + j;
        float a = x[0], e = x[half];
        if (h < nh + nkv) {
            rope_rotate(a, e, c, s, a, e);
            x[0] = a;
            x[half] = e;
        }
        if (h >= nh) {
            float* o = (h < nh + nkv ? S.k[b] + (long)(h - nh) * hd : S.v[b] + (long)(h - nh - nkv) * hd) + (long)pos * width + j;
            o[0] = a;
            o[half] = e;
        }
    }
}

// ------------------------------------------------------------------ KV append rows
// rows 0..nrows-1 of ksrc / vsrc (row stride src_ld) go to cache positions *len .. *len+nrows-1
__global__ void k_append_kv_rows(float* __restrict__ kbase, const float* __restrict__ ksrc, float* __restrict__ vbase,
                                 const float* __restrict__ vsrc, int src_ld, const int* __restrict__ len, int width,
                                 int max_seq, int nrows, int* status) {
    const int L = *len;
    if (L < 0 || L + nrows > max_seq) {
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(status, (int)LT_STATUS_KV_OVERFLOW);
        return;
    }
    const long total = (long)nrows * width;
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        const int r = (int)(i / width), c = (int)(i - (long)r * width);
        kbase[(long)(L + r) * width + c] = ksrc[(long)r * src_ld + c];
        vbase[(long)(L + r) * width + c] = vsrc[(long)r * src_ld + c];
    }
}
__global__ void k_add_len(int* len, int n, int max_seq) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        const int L = *len;
        if (L >= 0 && L + n <= max_seq) *len = L + n;
    }
}

// ------------------------------------------------------------------ silu * up -> quant, strided rows
// Four elements per thread, eight threads per block: bound by its 9 bytes per element and by the exponential and the
// division of silu.  A warp per block with one element per lane (k_silu_mul_quant_rows_lane) has four times
// the instructions around them: 2048 rows of 4864, 46.4 us, 21.0 with four.
__global__ void __launch_bounds__(256) k_silu_mul_quant_rows(const float* __restrict__ G, const float* __restrict__ U, int ld,
                                                             int8_t* __restrict__ Xq, __half* __restrict__ Xd, int K, int rows) {
    chain_release();
    chain_wait();
    const unsigned quads = (unsigned)K >> 2;
    const long i = (long)blockIdx.x * 256 + threadIdx.x;      // quad of elements, row-major
    const bool ok = i < (long)rows * quads;
    const long r = ok ? i / quads : 0;
    const long src = r * ld + (ok ? i - r * quads : 0) * 4;
    const float4 g = *(const float4*)(G + src), u = *(const float4*)(U + src);
    const float v[4] = {silu_mul(g.x, u.x), silu_mul(g.y, u.y), silu_mul(g.z, u.z), silu_mul(g.w, u.w)};
    __half d;
    const char4 q = quant_four(v, &d);
    if (!ok) return;
    ((char4*)Xq)[i] = q;
    if ((i & 7) == 0) Xd[i >> 3] = d;
}

// any alignment, and few blocks: a quarter of the chain of divisions (1 x 4864: 1.64 us, 1.75 with four; 150 x 896: 1.82, 2.11)
__global__ void k_silu_mul_quant_rows_lane(const float* __restrict__ G, const float* __restrict__ U, int ld,
                                           int8_t* __restrict__ Xq, __half* __restrict__ Xd, int K, int rows) {
    chain_release();
    chain_wait();
    const int nb = K >> 5;
    const long blk = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (blk >= (long)rows * nb) return;
    const int r = (int)(blk / nb), b = (int)(blk - (long)r * nb);
    const long src = (long)r * ld + (long)b * 32 + lane;
    const float v = silu_mul(G[src], U[src]);
    __half d;
    const int q = quant_lane(v, &d);
    Xq[(long)r * K + (long)b * 32 + lane] = (int8_t)q;
    if (lane == 0) Xd[(long)r * nb + b] = d;
}

// ------------------------------------------------------------------ causal attention over a chunk of rows
// Row r of the chunk is the query at cache position L0 + r, L0 = *len - nrows (the chunk's K/V rows
// are already appended), and sees L_r = L0 + r + 1 positions.  Per (row, head) the arithmetic is the
// one-token kernel's (lt_attn.cu): sequential-i fma scores, * scale, max, __expf, Z on 64 strided
// lanes + tree, left-fold V sum, / Z.
constexpr int PF_THREADS = 256;
constexpr int PF_KTILE = 128;            // K rows staged per tile: two threads per position

// What a row divides by.  A row none of whose scores reaches -1e30, the score of masked positions in the declared order (infinite and huge
// queries), has only zeros as probabilities; the declared kernel then counts its masked positions and returns zeros.
__device__ __forceinline__ float denominator(float z) { return z == 0.0f ? 1.0f : z; }

// The sequences of a launch.  One: its length on the device; several: their lengths after the append, from the host.  Together
// short prompts fill the SMs with blocks of 32 rows (three of 333: 87 us one after the other with 16 rows, 55 together).
struct AttnSeqs {
    const float *k[LT_ROW_SEQS], *v[LT_ROW_SEQS];
    const int* len;
    int total[LT_ROW_SEQS];
    __device__ __forceinline__ int length(int b) const { return len != nullptr ? *len : total[b]; }
};

template <int HD, int QT>
__global__ void __launch_bounds__(PF_THREADS, QT <= 8 ? 3 : 1)
k_attn_prefill(const float* __restrict__ Q, int q_ld, const float* __restrict__ K, const float* __restrict__ V,
               const int* __restrict__ len_ptr, float* __restrict__ OUT, int out_ld, int nh, int nkv, float scale,
               int nrows, int maxt, int* status) {
    extern __shared__ __align__(16) float pf_smem[];
    float* qs = pf_smem;                 // [QT][HD]
    float* red = qs + QT * HD;           // [QT][64]
    float* zs = red + QT * 64;           // [QT] max, then Z
    float* kt = zs + ((QT + 3) & ~3);    // [PF_KTILE][HD + 4] one tile of K rows (rows padded: conflict-free 16-byte reads)
    float* sc = kt + PF_KTILE * (HD + 4);   // [QT][ld], ld = maxt rounded up to 4 floats
    const int ld = (maxt + 3) & ~3;
    const int tid = threadIdx.x;
    const int h = blockIdx.y;
    const int r0 = blockIdx.x * QT;
    int Lafter = *len_ptr;
    if (Lafter < nrows || Lafter > maxt) {
        if (tid == 0) atomicOr(status, (int)LT_STATUS_BAD_LENGTH);
        return;
    }
    const int L0 = Lafter - nrows;
    const int nq = nrows - r0 < QT ? nrows - r0 : QT;   // query rows of this tile
    const int Lmax = L0 + r0 + nq;                      // positions the last row sees
    const int hk = h / (nh / nkv);

    for (int i = tid; i < QT * HD; i += PF_THREADS) {
        const int qi = i / HD, d = i - qi * HD;
        qs[i] = qi < nq ? Q[(long)(r0 + qi) * q_ld + (long)h * HD + d] : 0.0f;
    }
    __syncthreads();

    // scores: K rows go through shared memory in tiles of PF_KTILE positions (coalesced 16-byte asynchronous
    // copies; a thread reading its own row straight from global memory touches a new sector with every load).
    // A position of the tile is served by two threads, QT/2 queries each; each (row, query) score is the same
    // sequential-i fma chain as in the one-token kernel.
    constexpr int KST = HD + 4, QH = QT / 2;
    const int p = tid & (PF_KTILE - 1), qh = tid / PF_KTILE;
    for (int t0 = 0; t0 < Lmax; t0 += PF_KTILE) {
        const int nt = Lmax - t0 < PF_KTILE ? Lmax - t0 : PF_KTILE;
        for (int e = tid; e < nt * (HD / 4); e += PF_THREADS) {
            const int r = e / (HD / 4), c = e - r * (HD / 4);
            const float* src = K + ((long)(t0 + r) * nkv + hk) * HD + c * 4;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(kt + r * KST + c * 4)),
                         "l"(src) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (p < nt) {
            const int t = t0 + p;
            const float4* Kt = (const float4*)(kt + p * KST);
            float s[QH];
#pragma unroll
            for (int qi = 0; qi < QH; qi++) s[qi] = 0.0f;
#pragma unroll 4
            for (int i = 0; i < HD / 4; i++) {
                const float4 kk = Kt[i];
#pragma unroll
                for (int qi = 0; qi < QH; qi++) {
                    const float4 qq = ((const float4*)(qs + (qh * QH + qi) * HD))[i];
                    s[qi] = __fmaf_rn(qq.x, kk.x, s[qi]);
                    s[qi] = __fmaf_rn(qq.y, kk.y, s[qi]);
                    s[qi] = __fmaf_rn(qq.z, kk.z, s[qi]);
                    s[qi] = __fmaf_rn(qq.w, kk.w, s[qi]);
                }
            }
#pragma unroll
            for (int qi = 0; qi < QH; qi++) {
                const int q = qh * QH + qi;
                sc[q * ld + t] = t < L0 + r0 + q + 1 ? __fmul_rn(s[qi], scale) : -1e30f;
            }
        }
        __syncthreads();        // the tile is rewritten
    }

    // softmax per query row on the frozen 64-lane layout: 4 rows at a time, 64 threads each
    const int grp = tid >> 6, l64 = tid & 63;
    for (int qb = 0; qb < QT; qb += 4) {
        const int qi = qb + grp;
        float* row = sc + qi * ld;
        float m = -1e30f;
        for (int t = l64; t < Lmax; t += 64) m = fmaxf(m, row[t]);
        red[qi * 64 + l64] = m;
        __syncthreads();
        if (l64 < 32) {
            float v = fmaxf(red[qi * 64 + l64], red[qi * 64 + l64 + 32]);
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, s));
            if (l64 == 0) zs[qi] = v;
        }
        __syncthreads();
        const float mx = zs[qi];
        for (int t = l64; t < Lmax; t += 64) row[t] = __expf(__fsub_rn(row[t], mx));
        __syncthreads();
        float ls = 0.0f;
        for (int t = l64; t < Lmax; t += 64) ls = __fadd_rn(ls, row[t]);
        red[qi * 64 + l64] = ls;
        __syncthreads();
        if (l64 < 32) {
            float v = __fadd_rn(red[qi * 64 + l64], red[qi * 64 + l64 + 32]);
            v = warp_tree_sum(v);
            if (l64 == 0) zs[qi] = denominator(v);
        }
        __syncthreads();
    }

    // V sum: thread = (row group, two neighbouring output elements); a V row is read once per group as 8-byte
    // loads and serves the group's rows, so the loop is bound by its FMAs, not by loads
    constexpr int DV = 2;
    constexpr int TPG = HD / DV;             // threads per row group
    constexpr int NG = PF_THREADS / TPG;     // row groups
    constexpr int RPG = (QT + NG - 1) / NG;  // rows per group
    const int g = tid / TPG, d = (tid - g * TPG) * DV;
    float2 acc[RPG];
    int Lr[RPG];
#pragma unroll
    for (int k = 0; k < RPG; k++) {
        acc[k] = make_float2(0.0f, 0.0f);
        const int qi = g + k * NG;
        Lr[k] = qi < nq ? L0 + r0 + qi + 1 : 0;
    }
    const float* Vd = V + (long)hk * HD + d;
    const long vstride = (long)nkv * HD;
    // positions every row of the tile sees: four at a time, the probabilities as one 16-byte load
    const int Lcommon = (L0 + r0 + 1) & ~3;
    int t = 0;
    for (; t < Lcommon; t += 4) {
        const float2 v0 = *(const float2*)(Vd + (long)t * vstride), v1 = *(const float2*)(Vd + (long)(t + 1) * vstride);
        const float2 v2 = *(const float2*)(Vd + (long)(t + 2) * vstride), v3 = *(const float2*)(Vd + (long)(t + 3) * vstride);
#pragma unroll
        for (int k = 0; k < RPG; k++) {
            if (g + k * NG < QT) {
                const float4 pr = *(const float4*)(sc + (g + k * NG) * ld + t);
                acc[k].x = __fmaf_rn(pr.x, v0.x, acc[k].x); acc[k].y = __fmaf_rn(pr.x, v0.y, acc[k].y);
                acc[k].x = __fmaf_rn(pr.y, v1.x, acc[k].x); acc[k].y = __fmaf_rn(pr.y, v1.y, acc[k].y);
                acc[k].x = __fmaf_rn(pr.z, v2.x, acc[k].x); acc[k].y = __fmaf_rn(pr.z, v2.y, acc[k].y);
                acc[k].x = __fmaf_rn(pr.w, v3.x, acc[k].x); acc[k].y = __fmaf_rn(pr.w, v3.y, acc[k].y);
            }
        }
    }
    for (; t < Lmax; t++) {   // the causal edge: row by row
        const float2 v = *(const float2*)(Vd + (long)t * vstride);
#pragma unroll
        for (int k = 0; k < RPG; k++) {
            const int qi = g + k * NG;
            if (t < Lr[k]) {
                const float pr = sc[qi * ld + t];
                acc[k].x = __fmaf_rn(pr, v.x, acc[k].x);
                acc[k].y = __fmaf_rn(pr, v.y, acc[k].y);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < RPG; k++) {
        const int qi = g + k * NG;
        if (qi < nq) {
            const float z = zs[qi];
            *(float2*)(OUT + (long)(r0 + qi) * out_ld + (long)h * HD + d) = make_float2(__fdiv_rn(acc[k].x, z), __fdiv_rn(acc[k].y, z));
        }
    }
}

// ---- the same attention for 16 query rows per CTA (one CTA of 512 threads per SM).  A tile of K (then V) rows
// serves 16 query rows (half the L2 traffic of the 8-row kernel above), the next tile's asynchronous copy runs
// while this one is used (two buffers; the copies then cost ~1 k cycles per tile, barriers included, and nothing
// waits for them), and the first V tile is requested before the softmax.  What is left is shared-memory reads
// per fused multiply-add, so both folds are blocked in registers: a score thread owns two positions and four
// query rows (two K reads and four broadcast q reads per 32 FMAs), a V-sum thread two neighbouring output
// elements of two query rows.  Every (row, head) result is the one-token kernel's, bit for bit.
constexpr int PW_THREADS = 512;
constexpr int PW_QT = 16;
constexpr int PW_TILE = 128;             // positions per staged tile of K or V rows

template <int HD>
__global__ void __launch_bounds__(PW_THREADS, 1)
k_attn_prefill_wide(const float* __restrict__ Q, int q_ld, const __grid_constant__ AttnSeqs S, float* __restrict__ OUT, int out_ld, int nh,
                    int nkv, float scale, int nrows, int maxt, int* status) {
    constexpr int QT = PW_QT, KST = HD + 4;
    extern __shared__ __align__(16) float pf_smem[];
    float* qs = pf_smem;                     // [QT][HD]
    float* red = qs + QT * HD;               // [QT][64]
    float* zs = red + QT * 64;               // [QT] max, then Z
    float* tiles = zs + QT;                  // [2][PW_TILE][KST]
    float* sc = tiles + 2 * PW_TILE * KST;   // [QT][ld]
    const int ld = (maxt + 3) & ~3;
    const int tid = threadIdx.x;
    const int h = blockIdx.y;
    const int r0 = blockIdx.x * QT;
    const int seq = blockIdx.z, Lafter = S.length(seq);
    const float *K = S.k[seq], *V = S.v[seq];
    Q += (long)seq * nrows * q_ld;
    OUT += (long)seq * nrows * out_ld;
    if (Lafter < nrows || Lafter > maxt) {
        if (tid == 0) atomicOr(status, (int)LT_STATUS_BAD_LENGTH);
        return;
    }
    const int L0 = Lafter - nrows;
    const int nq = nrows - r0 < QT ? nrows - r0 : QT;   // query rows of this tile
    const int Lmax = L0 + r0 + nq;                      // positions the last row sees
    const int hk = h / (nh / nkv);
    const long rstride = (long)nkv * HD;                // floats between two positions of a cache

    auto copy_tile = [&](const float* base, int t0, float* dst) {     // positions [t0, t0 + PW_TILE) of head hk, one commit group
        const int nt = Lmax - t0 < PW_TILE ? Lmax - t0 : PW_TILE;
        const float* src = base + (long)hk * HD + (long)t0 * rstride;
        for (int e = tid; e < nt * (HD / 4); e += PW_THREADS) {
            const int r = e / (HD / 4), c = e - r * (HD / 4);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst + r * KST + c * 4)),
                         "l"(src + (long)r * rstride + c * 4) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    copy_tile(K, 0, tiles);
    for (int i = tid; i < QT * HD; i += PW_THREADS) {
        const int qi = i / HD, d = i - qi * HD;
        qs[i] = qi < nq ? Q[(long)(r0 + qi) * q_ld + (long)h * HD + d] : 0.0f;
    }

    // ---- scores: a thread owns two positions of the tile (p and p + 64) and four query rows: eight chains fed by two
    // 16-byte reads of K rows and four broadcast reads of q per four elements (half the shared-memory traffic per
    // fused multiply-add of one position per thread); 256 threads fold, all copy
    constexpr int QH = 4, PH = PW_TILE / 2;
    const int p = tid & (PH - 1), qh = tid / PH;
    for (int t0 = 0, buf = 0; t0 < Lmax; t0 += PW_TILE, buf ^= 1) {
        const bool more = t0 + PW_TILE < Lmax;
        if (more) copy_tile(K, t0 + PW_TILE, tiles + (buf ^ 1) * PW_TILE * KST);
        if (more) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                    // tile t0 has landed (and, first pass, the q rows are stored)
        const int nt = Lmax - t0 < PW_TILE ? Lmax - t0 : PW_TILE;
        if (qh < QT / QH && p < nt) {
            const bool two = p + PH < nt;
            const float4* Ka = (const float4*)(tiles + buf * PW_TILE * KST + p * KST);
            const float4* Kb = (const float4*)(tiles + buf * PW_TILE * KST + (two ? p + PH : p) * KST);
            const float4* Qt = (const float4*)(qs + qh * QH * HD);
            float sa[QH], sb[QH];
#pragma unroll
            for (int qi = 0; qi < QH; qi++) { sa[qi] = 0.0f; sb[qi] = 0.0f; }
#pragma unroll 4
            for (int i = 0; i < HD / 4; i++) {
                const float4 ka = Ka[i], kb = Kb[i];
                float4 qq[QH];
#pragma unroll
                for (int qi = 0; qi < QH; qi++) qq[qi] = Qt[qi * (HD / 4) + i];
#pragma unroll
                for (int qi = 0; qi < QH; qi++) { sa[qi] = __fmaf_rn(qq[qi].x, ka.x, sa[qi]); sb[qi] = __fmaf_rn(qq[qi].x, kb.x, sb[qi]); }
#pragma unroll
                for (int qi = 0; qi < QH; qi++) { sa[qi] = __fmaf_rn(qq[qi].y, ka.y, sa[qi]); sb[qi] = __fmaf_rn(qq[qi].y, kb.y, sb[qi]); }
#pragma unroll
                for (int qi = 0; qi < QH; qi++) { sa[qi] = __fmaf_rn(qq[qi].z, ka.z, sa[qi]); sb[qi] = __fmaf_rn(qq[qi].z, kb.z, sb[qi]); }
#pragma unroll
                for (int qi = 0; qi < QH; qi++) { sa[qi] = __fmaf_rn(qq[qi].w, ka.w, sa[qi]); sb[qi] = __fmaf_rn(qq[qi].w, kb.w, sb[qi]); }
            }
#pragma unroll
            for (int qi = 0; qi < QH; qi++) {
                const int q = qh * QH + qi;
                const int ta = t0 + p, tb2 = ta + PH;
                sc[q * ld + ta] = ta < L0 + r0 + q + 1 ? __fmul_rn(sa[qi], scale) : -1e30f;
                if (two) sc[q * ld + tb2] = tb2 < L0 + r0 + q + 1 ? __fmul_rn(sb[qi], scale) : -1e30f;
            }
        }
        __syncthreads();                    // the tile may be overwritten, the scores are visible
    }
    // the first V tile travels while the softmax runs
    copy_tile(V, 0, tiles);

    // ---- softmax per query row on the frozen 64-lane layout: 8 rows at a time, 64 threads each
    const int grp = tid >> 6, l64 = tid & 63;
    for (int qb = 0; qb < QT; qb += PW_THREADS / 64) {
        const int qi = qb + grp;
        float* row = sc + qi * ld;
        float m = -1e30f;
        for (int t = l64; t < Lmax; t += 64) m = fmaxf(m, row[t]);
        red[qi * 64 + l64] = m;
        __syncthreads();
        if (l64 < 32) {
            float v = fmaxf(red[qi * 64 + l64], red[qi * 64 + l64 + 32]);
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, s));
            if (l64 == 0) zs[qi] = v;
        }
        __syncthreads();
        const float mx = zs[qi];
        float ls = 0.0f;
        for (int t = l64; t < Lmax; t += 64) {      // a lane sums what it has just written: no barrier in between
            const float e = __expf(__fsub_rn(row[t], mx));
            row[t] = e;
            ls = __fadd_rn(ls, e);
        }
        red[qi * 64 + l64] = ls;
        __syncthreads();
        if (l64 < 32) {
            float v = __fadd_rn(red[qi * 64 + l64], red[qi * 64 + l64 + 32]);
            v = warp_tree_sum(v);
            if (l64 == 0) zs[qi] = denominator(v);
        }
        __syncthreads();
    }

    // ---- V sum: thread = (group of two query rows, two neighbouring output elements); 256 threads fold, all copy
    constexpr int DV = 2, TPG = HD / DV, RPG = 2, NG = QT / RPG;
    static_assert(NG * TPG <= PW_THREADS, "row groups");
    const int g = tid / TPG, d = (tid - g * TPG) * DV;
    const bool folds = g < NG;
    float2 acc[RPG];
    int Lr[RPG];
#pragma unroll
    for (int k = 0; k < RPG; k++) {
        acc[k] = make_float2(0.0f, 0.0f);
        const int qi = g * RPG + k;
        Lr[k] = (folds && qi < nq) ? L0 + r0 + qi + 1 : 0;
    }
    // positions every row of the tile sees are folded four at a time, the probabilities as one 16-byte read
    const int Lcommon = (L0 + r0 + 1) & ~3;
    for (int t0 = 0, buf = 0; t0 < Lmax; t0 += PW_TILE, buf ^= 1) {
        const bool more = t0 + PW_TILE < Lmax;
        if (more) copy_tile(V, t0 + PW_TILE, tiles + (buf ^ 1) * PW_TILE * KST);
        if (more) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (folds) {
            const float* vt = tiles + buf * PW_TILE * KST + d;
            const float* pr0 = sc + (g * RPG) * ld;
            const int te = more ? t0 + PW_TILE : Lmax;
            const int tv = (te < Lcommon ? te : Lcommon) & ~3;
            int t = t0;
            for (; t + 4 <= tv; t += 4) {
                float2 v[4];
                float4 pr[RPG];
#pragma unroll
                for (int j = 0; j < 4; j++) v[j] = *(const float2*)(vt + (t + j - t0) * KST);
#pragma unroll
                for (int k = 0; k < RPG; k++) pr[k] = *(const float4*)(pr0 + k * ld + t);
#pragma unroll
                for (int k = 0; k < RPG; k++) { acc[k].x = __fmaf_rn(pr[k].x, v[0].x, acc[k].x); acc[k].y = __fmaf_rn(pr[k].x, v[0].y, acc[k].y); }
#pragma unroll
                for (int k = 0; k < RPG; k++) { acc[k].x = __fmaf_rn(pr[k].y, v[1].x, acc[k].x); acc[k].y = __fmaf_rn(pr[k].y, v[1].y, acc[k].y); }
#pragma unroll
                for (int k = 0; k < RPG; k++) { acc[k].x = __fmaf_rn(pr[k].z, v[2].x, acc[k].x); acc[k].y = __fmaf_rn(pr[k].z, v[2].y, acc[k].y); }
#pragma unroll
                for (int k = 0; k < RPG; k++) { acc[k].x = __fmaf_rn(pr[k].w, v[3].x, acc[k].x); acc[k].y = __fmaf_rn(pr[k].w, v[3].y, acc[k].y); }
            }
            for (; t < te; t++) {   // the causal edge: row by row
                const float2 v = *(const float2*)(vt + (t - t0) * KST);
#pragma unroll
                for (int k = 0; k < RPG; k++) {
                    if (t < Lr[k]) {
                        const float pr = pr0[k * ld + t];
                        acc[k].x = __fmaf_rn(pr, v.x, acc[k].x);
                        acc[k].y = __fmaf_rn(pr, v.y, acc[k].y);
                    }
                }
            }
        }
        __syncthreads();                    // the tile may be overwritten
    }
#pragma unroll
    for (int k = 0; k < RPG; k++) {
        const int qi = g * RPG + k;
        if (folds && qi < nq) {
            const float z = zs[qi];
            *(float2*)(OUT + (long)(r0 + qi) * out_ld + (long)h * HD + d) = make_float2(__fdiv_rn(acc[k].x, z), __fdiv_rn(acc[k].y, z));
        }
    }
}

template <int HD>
static size_t attn_prefill_wide_smem(int maxt) {
    return ((size_t)PW_QT * HD + PW_QT * 64 + PW_QT + (size_t)2 * PW_TILE * (HD + 4) + (size_t)PW_QT * ((maxt + 3) & ~3)) * sizeof(float);
}

template <int HD>
static int launch_attn_prefill_wide(const float* Q, int q_ld, const AttnSeqs& S, int nseq, float* OUT, int out_ld, int nh, int nkv,
                                    float scale, int nrows, int maxt, cudaStream_t s) {
    int* st = device_status_ptr();
    LT_REQUIRE(st != nullptr, "lt_attn_prefill: status word unavailable");
    const size_t smem = attn_prefill_wide_smem<HD>(maxt);
    static PerDeviceOnce attr_once;
    if (attr_once.first()) {
        LT_CUDA(cudaFuncSetAttribute(k_attn_prefill_wide<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    }
    dim3 grid((nrows + PW_QT - 1) / PW_QT, nh, nseq);
    k_attn_prefill_wide<HD><<<grid, PW_THREADS, smem, s>>>(Q, q_ld, S, OUT, out_ld, nh, nkv, scale, nrows, maxt, st);
    return check_launch("lt_attn_prefill");
}

// ---- the same attention for long chunks: 32 query rows per CTA of 128 threads, as register-blocked products over tiles
// of 64 positions.  A score is a chain over d and an output a chain over positions, but different scores and outputs are
// independent, so both are halves of a blocked fp32 product whose inner loop runs in the declared order.  What the
// 16-row form above spends its time on is operand reads (6 of 16 bytes per 32 multiply-adds, 256 of 512 threads
// folding, one CTA per SM, phases between barriers).  Here a thread owns 4 rows x 4 positions, then 4 rows x HD / 16
// elements: 8 reads, 4 of them nearly broadcasts, per 64 multiply-adds, and CTAs overlap on an SM (four with heads of 64,
// two with heads of 128: 52 and 93 KB of shared memory).  The row maxima come first, by bounds from the tensor
// cores: no SM holds 32 rows of scores beside the tiles, and nothing depends on Lmax.  A row's 64 softmax lanes are the 64 positions of
// a tile, so the lane sums of the denominator stay in the registers of the threads that make the probabilities.  Bound by the operand reads (twice the clocks of the
// multiply-adds) and issue slots of its two exact products of Lmax^2 / 2 x HD per head and by the uneven lengths of the rows.
// 2048 positions: 14 heads on 2 of 64: 505 us with 16 rows, now 314; 32 heads on 8 of 128: 3273, now 1273.
// (64 rows per CTA, 8 x 4 per thread: 444; the 448 CTAs are all resident at once and share the SMs unevenly.)
constexpr int PB_TILE = 64;
constexpr int PREFILL_MAXT = 12000;      // positions that the entry points take
static_assert(PREFILL_MAXT <= PB_TILE * 2048, "a position's place within its thread has 13 bits");

template <int HD, int QT>
struct PrefillBlock {
    static constexpr int THREADS = 128;
    static constexpr int ST = HD + 4;                    // floats between rows: conflict-free 16-byte reads
    static constexpr int PST = PB_TILE + 4;
    static constexpr int SMEM = (QT * ST + 2 * PB_TILE * ST + QT * PST + QT) * 4;
};

template <int HD, int QT>
__global__ void __launch_bounds__(PrefillBlock<HD, QT>::THREADS, HD == 64 ? 4 : 2)
k_attn_prefill_block(const float* __restrict__ Q, int q_ld, const __grid_constant__ AttnSeqs S, int nseq, float* __restrict__ OUT, int out_ld,
                     int nh, int nkv, float scale, int nrows, int maxt, int* status) {
    using B = PrefillBlock<HD, QT>;
    constexpr int PB_THREADS = B::THREADS, ST = B::ST, PST = B::PST, MQ = QT * 16 / PB_THREADS, ND = HD / 64;
    extern __shared__ __align__(16) float pf_smem[];
    float* qs = pf_smem;                     // [QT][ST]
    float* tk = qs + QT * ST;                // [PB_TILE][ST]  K
    float* tv = tk + PB_TILE * ST;           // [PB_TILE][ST]  V (the other K buffer while the maxima are found)
    float* ps = tv + PB_TILE * ST;           // [QT][PST] probabilities of a tile, at the end the lane sums
    float* zs = ps + QT * PST;               // [QT]
    const int tid = threadIdx.x, n = tid & 15, m = tid >> 4;
    const int h = blockIdx.x % nh;
    const int step = (int)blockIdx.x / nh, seq = step % nseq;
    const int r0 = ((int)gridDim.x / nh / nseq - 1 - step / nseq) * QT;       // the longest rows first
    const int Lafter = S.length(seq);
    const float *K = S.k[seq], *V = S.v[seq];
    Q += (long)seq * nrows * q_ld;
    OUT += (long)seq * nrows * out_ld;
    if (Lafter < nrows || Lafter > maxt) {
        if (tid == 0) atomicOr(status, (int)LT_STATUS_BAD_LENGTH);
        return;
    }
    const int L0 = Lafter - nrows;
    const int nq = nrows - r0 < QT ? nrows - r0 : QT;
    const int Lmax = L0 + r0 + nq;
    const int hk = h / (nh / nkv);
    const long rstride = (long)nkv * HD;

    auto copy_tile = [&](const float* base, int t0, float* dst) {     // positions [t0, t0 + 64) of head hk; zeros from Lmax on
        const float* src = base + (long)hk * HD + (long)t0 * rstride;
#pragma unroll 4
        for (int e = tid; e < PB_TILE * (HD / 4); e += PB_THREADS) {
            const int r = e / (HD / 4), c = e - r * (HD / 4);
            const bool ok = t0 + r < Lmax;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst + r * ST + c * 4)),
                         "l"(ok ? src + (long)r * rstride + c * 4 : base), "r"(ok ? 16 : 0)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // scores of rows m * MQ + i and positions t0 + n + 16 j of a K tile, not yet scaled
    auto scores = [&](const float* kt, float (&s)[MQ][4]) {
#pragma unroll
        for (int i = 0; i < MQ; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) s[i][j] = 0.0f;
        const float4* K4 = (const float4*)(kt + n * ST);
        const float4* Q4 = (const float4*)(qs + m * MQ * ST);
#pragma unroll 4
        for (int d = 0; d < HD / 4; d++) {
            float4 k[4], q[MQ];
#pragma unroll
            for (int j = 0; j < 4; j++) k[j] = K4[j * 16 * (ST / 4) + d];
#pragma unroll
            for (int i = 0; i < MQ; i++) q[i] = Q4[i * (ST / 4) + d];
#pragma unroll
            for (int i = 0; i < MQ; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) s[i][j] = __fmaf_rn(q[i].x, k[j].x, s[i][j]);
#pragma unroll
            for (int i = 0; i < MQ; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) s[i][j] = __fmaf_rn(q[i].y, k[j].y, s[i][j]);
#pragma unroll
            for (int i = 0; i < MQ; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) s[i][j] = __fmaf_rn(q[i].z, k[j].z, s[i][j]);
#pragma unroll
            for (int i = 0; i < MQ; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) s[i][j] = __fmaf_rn(q[i].w, k[j].w, s[i][j]);
        }
    };

    copy_tile(K, 0, tk);
    for (int e = tid; e < QT * (HD / 4); e += PB_THREADS) {
        const int r = e / (HD / 4), c = e - r * (HD / 4);
        *(float4*)(qs + r * ST + c * 4) =
            r < nq ? *(const float4*)(Q + (long)(r0 + r) * q_ld + (long)h * HD + c * 4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    int lim[MQ];                             // positions that row i sees
#pragma unroll
    for (int i = 0; i < MQ; i++) lim[i] = L0 + r0 + m * MQ + i + 1;

    // ---- row maxima.  Only the greatest score of a row is wanted here, and it need be exact only there: fp16 products on the
    // tensor cores (mma: a sixteenth of the shared-memory reads of the blocked product) are within eps of every score, so product +
    // eps bounds a score from above.  With u = 2^-11, the largest relative error of a rounding to 11 bits, and 2^-25, the largest
    // error of one to a subnormal fp16, the product of the rounded rows is off by at most
    //     2^-10 (1 + 2^-12) |q| |k| + 2^-25 sqrt(HD) (|q| + |k|) (1 + u) + 2^-50 HD;
    // its sums and the declared chain's add less than 2^-14 |q| |k|, and the place below, which takes 13 bits of the bound, 2^-10 of
    // it.  eps = 2.25 x 2^-10 (|q| + 2^-12) (|k| + 2^-12) |scale| is more than all of them (2.07 x 2^-10 |q| |k|; 2^-25 sqrt(128) = 0.63
    // x 2.25 x 2^-22).  The norms' own rounding is below 2^-16 of eps, and 1e-37 covers products that underflow.
    // A thread sees a sixteenth of a row's positions and keeps the three greatest bounds, the place in the low 13 bits of each.  The
    // declared chain of every warp's greatest gives a score that the maximum reaches at least; what else may reach it (one or two of
    // a row, from the first two of a thread) is folded too.  Where a third may, or many do (rows of equal scores), or eps is no bound
    // (norms at the end of fp16 or beyond, or not finite), the blocked product finds the maxima.
    // 2048 positions, us, with the blocked product alone and so: 14 heads of 64 350 and 314, 32 heads of 128 1550 and 1273; with keys
    // whose bias is three times their deviation 349 and 314, 1549 and 1288; eight times 349 and 331, 1550 and 1401; twenty times 350
    // and 369, 1547 and 1558; equal keys 350 and 350, 1550 and 1558.  (bf16 needs a bound four times as wide; products in tf32:
    // 406; candidates found by a second walk over K: 350.)
    float mx[MQ];
#pragma unroll
    for (int i = 0; i < MQ; i++) mx[i] = -1e30f;
    bool blocked;
    {
        static_assert(QT == 32 && PB_THREADS == 128 && PB_TILE == 64, "a warp takes 16 positions of a tile for 32 rows");
        constexpr int NCAND = 2 * PB_THREADS;    // one for each warp and row, as many others
        const int w = tid >> 5, g = (tid & 31) >> 2, t4 = tid & 3;
        int* mk = (int*)ps;                      // [QT] greatest exact score, as an ordered integer
        int* ncand = mk + QT;
        int* list = ncand + 4;                   // [NCAND] candidates: position * 32 + row
        static_assert(QT + 4 + NCAND <= QT * PST, "candidates beside the maxima");
        auto ordered = [](int v) { return v ^ ((v >> 31) & 0x7fffffff); };
        auto fp16 = [](float lo, float hi) {
            unsigned r;
            asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
            return r;
        };
        auto chain = [&](int at) {
            const int r = at & 31;
            const float4* q4 = (const float4*)(qs + r * ST);
            const float4* k4 = (const float4*)(K + (long)hk * HD + (long)(at >> 5) * rstride);
            float v = 0.0f;
#pragma unroll 8
            for (int d = 0; d < HD / 4; d++) {
                const float4 q = q4[d], k = __ldg(k4 + d);
                v = __fmaf_rn(q.x, k.x, v); v = __fmaf_rn(q.y, k.y, v);
                v = __fmaf_rn(q.z, k.z, v); v = __fmaf_rn(q.w, k.w, v);
            }
            atomicMax(mk + r, ordered(__float_as_int(__fmul_rn(v, scale))));
        };
        list[tid] = -1;
        if (tid < QT) mk[tid] = ordered(__float_as_int(-1e30f));
        if (tid == 0) *ncand = 0;
        __syncthreads();                         // the q rows are stored
        // Fragments: thread t4 of a row's four holds elements 16 c + 4 t4 .. + 3 (a sum may take the elements in any order as
        // long as both operands agree).
        unsigned qa[HD / 16][2][2][2];           // [16 elements][16 rows][row g or g + 8][pair]
        float qn[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // squared norms of rows g + 8 i, then eps / |k|
#pragma unroll
        for (int c = 0; c < HD / 16; c++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float4 q = *(const float4*)(qs + (g + 8 * i) * ST + 16 * c + 4 * t4);
                qn[i] += q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w;
                qa[c][i >> 1][i & 1][0] = fp16(q.x, q.y);
                qa[c][i >> 1][i & 1][1] = fp16(q.z, q.w);
            }
        float top[4][3];                         // rows g + 8 i
        bool bad = false;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            qn[i] += __shfl_xor_sync(0xffffffffu, qn[i], 1);
            qn[i] += __shfl_xor_sync(0xffffffffu, qn[i], 2);
            bad = bad || !(qn[i] < 4e9f);        // no element beyond 63245
            qn[i] = (sqrtf(qn[i]) + 0x1p-12f) * fabsf(scale) * (2.25f / 1024.0f);
            bad = bad || !(qn[i] < 1e14f);
            top[i][0] = top[i][1] = top[i][2] = -1e38f;
        }
        float kg = 0.0f;                         // norm of a key of the last tile
        int t0 = 0, buf = 0;
#pragma unroll 1
        for (int end = 2 * PB_TILE < Lmax ? 2 * PB_TILE : Lmax;; end = Lmax) {
#pragma unroll 1
            for (; t0 < end; t0 += PB_TILE, buf ^= 1) {
                if (t0 + PB_TILE < Lmax) {
                    copy_tile(K, t0 + PB_TILE, buf ? tk : tv);
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                } else {
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                }
                __syncthreads();
                const float* kt = (buf ? tv : tk) + (w * 16 + g) * ST + 4 * t4;
                const bool edge = t0 + PB_TILE > L0 + r0 + 1 || nq < QT;
                const int tp = t0 + w * 16 + 2 * t4 - (L0 + r0 + g);
#pragma unroll
                for (int y = 0; y < 2; y++) {        // eight positions
                    float c[2][4], k2 = 0.0f;
#pragma unroll
                    for (int x = 0; x < 2; x++)
#pragma unroll
                        for (int e = 0; e < 4; e++) c[x][e] = 0.0f;
#pragma unroll
                    for (int cc = 0; cc < HD / 16; cc++) {
                        const float4 k = *(const float4*)(kt + y * 8 * ST + 16 * cc);
                        k2 += k.x * k.x + k.y * k.y + k.z * k.z + k.w * k.w;
                        const unsigned k0 = fp16(k.x, k.y), k1 = fp16(k.z, k.w);
#pragma unroll
                        for (int x = 0; x < 2; x++)
                            asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                                : "+f"(c[x][0]), "+f"(c[x][1]), "+f"(c[x][2]), "+f"(c[x][3])
                                : "r"(qa[cc][x][0][0]), "r"(qa[cc][x][1][0]), "r"(qa[cc][x][0][1]), "r"(qa[cc][x][1][1]), "r"(k0), "r"(k1));
                    }
                    k2 += __shfl_xor_sync(0xffffffffu, k2, 1);
                    k2 += __shfl_xor_sync(0xffffffffu, k2, 2);
                    bad = bad || !(k2 < 4e9f);
                    kg = sqrtf(k2) + 0x1p-12f;       // of position g; the products are those of positions 2 t4 and 2 t4 + 1
                    const float kn[2] = {__shfl_sync(0xffffffffu, kg, 8 * t4), __shfl_sync(0xffffffffu, kg, 8 * t4 + 4)};
#pragma unroll
                    for (int x = 0; x < 2; x++)
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const int i = 2 * x + (e >> 1);
                            float v = __fmaf_rn(c[x][e], scale, __fmaf_rn(qn[i], kn[e & 1], 1e-37f));
                            if (edge && !(tp + 8 * y + (e & 1) <= 8 * i && g + 8 * i < nq)) v = -1e38f;
                            v = __int_as_float((__float_as_int(v) & ~0x1fff) | (t0 / PB_TILE * 4 + 2 * y + (e & 1)));
                            float(&a)[3] = top[i];
                            const float d0 = fminf(a[0], v);
                            a[0] = fmaxf(a[0], v);
                            const float d1 = fminf(a[1], d0);
                            a[1] = fmaxf(a[1], d0);
                            a[2] = fmaxf(a[2], d1);
                        }
                }
                __syncthreads();                     // the tile may be replaced
            }
            if (end == Lmax) break;
            // Keys much alike, beside their lengths, leave too many in the end.  Where a 32nd of the threads have a third of their eight
            // positions so far within reach of the warp's first (one of a thread's rows is asked; all four cost 2 us of code), the
            // search ends here, and what it took is a few per cent.
            float v = fmaxf(top[0][0], __shfl_xor_sync(0xffffffffu, top[0][0], 1));
            v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
            const bool near = bad || (top[0][2] > -9e37f && top[0][2] >= v - 2.0f * qn[0] * kg);
            if (__syncthreads_count(near) >= PB_THREADS / 32) {
                bad = true;
                break;
            }
        }
        auto position = [&](float v) {
            const int place = __float_as_int(v) & 0x1fff;
            return (place >> 2) * PB_TILE + w * 16 + (place & 2) * 4 + 2 * t4 + (place & 1);
        };
        // the greatest bound of the warp, where it sees a position of the row at all (of several threads with it, one)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float v = fmaxf(top[i][0], __shfl_xor_sync(0xffffffffu, top[i][0], 1));
            v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
            if (top[i][0] == v && v > -9e37f) list[w * QT + g + 8 * i] = position(v) * 32 + g + 8 * i;
        }
        blocked = __syncthreads_or(bad);
        if (!blocked) {
            if (list[tid] >= 0) chain(list[tid]);
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float least = __int_as_float(ordered(mk[g + 8 * i]));
                bad = bad || top[i][2] >= least;
#pragma unroll
                for (int j = 0; j < 2; j++)
                    if (top[i][j] >= least && !(j == 0 && list[w * QT + g + 8 * i] == position(top[i][0]) * 32 + g + 8 * i)) {
                        const int at = atomicAdd(ncand, 1);
                        if (at < NCAND - PB_THREADS) list[PB_THREADS + at] = position(top[i][j]) * 32 + g + 8 * i;
                    }
            }
            blocked = __syncthreads_or(bad) || *ncand > NCAND - PB_THREADS;
        }
        if (!blocked) {
            if (tid < *ncand) chain(list[PB_THREADS + tid]);
            __syncthreads();
#pragma unroll
            for (int i = 0; i < MQ; i++) mx[i] = fmaxf(mx[i], __int_as_float(ordered(mk[m * MQ + i])));
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");     // a tile may be on its way to where the first one goes
            copy_tile(K, 0, tk);
        }
    }
    for (int t0 = 0, buf = 0; blocked && t0 < Lmax; t0 += PB_TILE, buf ^= 1) {
        if (t0 + PB_TILE < Lmax) {
            copy_tile(K, t0 + PB_TILE, buf ? tk : tv);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        float s[MQ][4];
        scores(buf ? tv : tk, s);
#pragma unroll
        for (int i = 0; i < MQ; i++)
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (t0 + n + 16 * j < lim[i]) mx[i] = fmaxf(mx[i], __fmul_rn(s[i][j], scale));
        __syncthreads();
    }
    copy_tile(K, 0, tk);
    copy_tile(V, 0, tv);
#pragma unroll
    for (int i = 0; i < MQ; i++)
#pragma unroll
        for (int x = 8; x > 0; x >>= 1) mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], x));

    // ---- probabilities, lane sums of the denominator, V sum
    float z[MQ][4], acc[ND][MQ][4];
#pragma unroll
    for (int i = 0; i < MQ; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            z[i][j] = 0.0f;
#pragma unroll
            for (int g = 0; g < ND; g++) acc[g][i][j] = 0.0f;
        }
    for (int t0 = 0; t0 < Lmax; t0 += PB_TILE) {
        const bool more = t0 + PB_TILE < Lmax;
        asm volatile("cp.async.wait_group 1;" ::: "memory");      // K of this tile; V may be on its way
        __syncthreads();
        {
            float s[MQ][4];
            scores(tk, s);
#pragma unroll
            for (int i = 0; i < MQ; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float e = t0 + n + 16 * j < lim[i] ? __expf(__fsub_rn(__fmul_rn(s[i][j], scale), mx[i])) : 0.0f;
                    z[i][j] = __fadd_rn(z[i][j], e);
                    ps[(m * MQ + i) * PST + n + 16 * j] = e;
                }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                          // probabilities and V are there, K may be replaced
        if (more) copy_tile(K, t0 + PB_TILE, tk);
        const float* pr = ps + m * MQ * PST;
        if (t0 + PB_TILE <= L0 + r0 + 1) {                        // every row sees the whole tile
#pragma unroll 2
            for (int t = 0; t < PB_TILE; t += 4) {
                float4 p[MQ];
#pragma unroll
                for (int i = 0; i < MQ; i++) p[i] = *(const float4*)(pr + i * PST + t);
#pragma unroll
                for (int g = 0; g < ND; g++) {
                    float4 v[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) v[j] = *(const float4*)(tv + (t + j) * ST + g * 64 + n * 4);
#pragma unroll
                    for (int j = 0; j < 4; j++)
#pragma unroll
                        for (int i = 0; i < MQ; i++) {
                            const float w = j == 0 ? p[i].x : (j == 1 ? p[i].y : (j == 2 ? p[i].z : p[i].w));
                            acc[g][i][0] = __fmaf_rn(w, v[j].x, acc[g][i][0]);
                            acc[g][i][1] = __fmaf_rn(w, v[j].y, acc[g][i][1]);
                            acc[g][i][2] = __fmaf_rn(w, v[j].z, acc[g][i][2]);
                            acc[g][i][3] = __fmaf_rn(w, v[j].w, acc[g][i][3]);
                        }
                }
            }
        } else {                                                  // the causal edge: a row stops at its own position
            const int te = more ? PB_TILE : Lmax - t0;
            for (int t = 0; t < te; t++) {
#pragma unroll
                for (int g = 0; g < ND; g++) {
                    const float4 v = *(const float4*)(tv + t * ST + g * 64 + n * 4);
#pragma unroll
                    for (int i = 0; i < MQ; i++)
                        if (t0 + t < lim[i]) {
                            const float w = pr[i * PST + t];
                            acc[g][i][0] = __fmaf_rn(w, v.x, acc[g][i][0]);
                            acc[g][i][1] = __fmaf_rn(w, v.y, acc[g][i][1]);
                            acc[g][i][2] = __fmaf_rn(w, v.z, acc[g][i][2]);
                            acc[g][i][3] = __fmaf_rn(w, v.w, acc[g][i][3]);
                        }
                }
            }
        }
        __syncthreads();                                          // V and the probabilities may be replaced
        if (more) copy_tile(V, t0 + PB_TILE, tv);
    }

    // ---- denominator: 64 lanes of a row, then the tree
#pragma unroll
    for (int i = 0; i < MQ; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) ps[(m * MQ + i) * PST + n + 16 * j] = z[i][j];
    __syncthreads();
    for (int r = tid >> 5; r < QT; r += PB_THREADS / 32) {
        const float v = warp_tree_sum(__fadd_rn(ps[r * PST + (tid & 31)], ps[r * PST + (tid & 31) + 32]));
        if ((tid & 31) == 0) zs[r] = denominator(v);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MQ; i++) {
        const int r = m * MQ + i;
        if (r >= nq) continue;
        const float zr = zs[r];
#pragma unroll
        for (int g = 0; g < ND; g++) {
            float* o = OUT + (long)(r0 + r) * out_ld + (long)h * HD + g * 64 + n * 4;
            ((float2*)o)[0] = make_float2(__fdiv_rn(acc[g][i][0], zr), __fdiv_rn(acc[g][i][1], zr));
            ((float2*)o)[1] = make_float2(__fdiv_rn(acc[g][i][2], zr), __fdiv_rn(acc[g][i][3], zr));
        }
    }
}

template <int HD, int QT>
static int launch_attn_prefill_block(const float* Q, int q_ld, const AttnSeqs& S, int nseq, float* OUT, int out_ld, int nh, int nkv,
                                     float scale, int nrows, int maxt, cudaStream_t s) {
    int* st = device_status_ptr();
    LT_REQUIRE(st != nullptr, "lt_attn_prefill: status word unavailable");
    constexpr int smem = PrefillBlock<HD, QT>::SMEM;
    static PerDeviceOnce attr_once;
    if (attr_once.first()) {
        LT_CUDA(cudaFuncSetAttribute(k_attn_prefill_block<HD, QT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    }
    k_attn_prefill_block<HD, QT><<<(nrows + QT - 1) / QT * nh * nseq, PrefillBlock<HD, QT>::THREADS, smem, s>>>(
        Q, q_ld, S, nseq, OUT, out_ld, nh, nkv, scale, nrows, maxt, st);
    return check_launch("lt_attn_prefill");
}

template <int HD, int QT>
static int launch_attn_prefill(const float* Q, int q_ld, const float* K, const float* V, const int* len, float* OUT,
                               int out_ld, int nh, int nkv, float scale, int nrows, int maxt, cudaStream_t s) {
    int* st = device_status_ptr();
    LT_REQUIRE(st != nullptr, "lt_attn_prefill: status word unavailable");
    const size_t smem = ((size_t)QT * HD + QT * 64 + ((QT + 3) & ~3) + (size_t)PF_KTILE * (HD + 4) +
                         (size_t)QT * ((maxt + 3) & ~3)) * sizeof(float);
    LT_REQUIRE(smem <= 200 * 1024, "lt_attn_prefill: maxt=%d needs %zu bytes of shared memory", maxt, smem);
    static PerDeviceOnce attr_once;
    if (attr_once.first()) {
        LT_CUDA(cudaFuncSetAttribute(k_attn_prefill<HD, QT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    }
    dim3 grid((nrows + QT - 1) / QT, nh);
    k_attn_prefill<HD, QT><<<grid, PF_THREADS, smem, s>>>(Q, q_ld, K, V, len, OUT, out_ld, nh, nkv, scale, nrows, maxt,
                                                         st);
    return check_launch("lt_attn_prefill");
}

// The forms that take several sequences at once, LT_ERR_UNSUPPORTED where none fits
template <int HD>
static int pick_attn_prefill_rows(const float* Q, int q_ld, const AttnSeqs& S, int nseq, float* OUT, int out_ld, int nh, int nkv,
                                  float scale, int nrows, int maxt, cudaStream_t s) {
    bool aligned = true;
    for (int b = 0; b < nseq; b++) aligned = aligned && aligned16(S.v[b]);
    if (nrows >= 32 && aligned) {
        // 32 rows per CTA from two CTAs (heads of 64) or 9/4 (heads of 128) for each SM on; below, smaller tiles fill the SMs
        // better.  us with 16 and with 32 rows per CTA: 14 heads of 64, 333 rows (154 CTAs) 31 and 36, 500 (224) 52 and 60, 600 (266)
        // 67 and 62, 700 (308) 84 and 79, 850 (378) 115 and 97 (with equal keys, whose maxima the blocked product finds, 700 rows 91, 850
        // rows 113); of 128, 16 heads, 600 rows (304) 121 and 125, 32 heads, 300 rows (320) 74 and 67, 400 behind 700 positions (416)
        // 358 and 346.
        if ((long)((nrows + 31) / 32) * nh * nseq * 4 >= (HD == 64 ? 8L : 9L) * sm_count())
            return launch_attn_prefill_block<HD, 32>(Q, q_ld, S, nseq, OUT, out_ld, nh, nkv, scale, nrows, maxt, s);
        // ... where the score rows of 16 queries fit one SM beside double-buffered tiles
        if (attn_prefill_wide_smem<HD>(maxt) <= 227 * 1024)
            return launch_attn_prefill_wide<HD>(Q, q_ld, S, nseq, OUT, out_ld, nh, nkv, scale, nrows, maxt, s);
    }
    return LT_ERR_UNSUPPORTED;
}

template <int HD>
static int pick_attn_prefill(const float* Q, int q_ld, const float* K, const float* V, const int* len, float* OUT,
                             int out_ld, int nh, int nkv, float scale, int nrows, int maxt, cudaStream_t s) {
    AttnSeqs S = {};
    S.k[0] = K; S.v[0] = V; S.len = len;
    const int rc = pick_attn_prefill_rows<HD>(Q, q_ld, S, 1, OUT, out_ld, nh, nkv, scale, nrows, maxt, s);
    if (rc != LT_ERR_UNSUPPORTED) return rc;
    // query rows per tile: 8 while three CTAs of score rows fit an SM (the V sum and the softmax are
    // chains of dependent operations, resident warps hide them), else 4; 16 only for short chunks
    const size_t per_row = (size_t)((maxt + 3) & ~3) + HD + 65;
    const size_t tile = (size_t)PF_KTILE * (HD + 4) * sizeof(float);
    if (16 * per_row * sizeof(float) + tile <= 72 * 1024)
        return launch_attn_prefill<HD, 16>(Q, q_ld, K, V, len, OUT, out_ld, nh, nkv, scale, nrows, maxt, s);
    if (8 * per_row * sizeof(float) + tile <= 110 * 1024 || 4 * per_row * sizeof(float) + tile > 200 * 1024 / 2)
        return launch_attn_prefill<HD, 8>(Q, q_ld, K, V, len, OUT, out_ld, nh, nkv, scale, nrows, maxt, s);
    return launch_attn_prefill<HD, 4>(Q, q_ld, K, V, len, OUT, out_ld, nh, nkv, scale, nrows, maxt, s);
}

}  // namespace lt

using namespace lt;

extern "C" int lt_embed_q8_rows(const int8_t* Wq, const uint16_t* Wd, const int* toks, float* out, int E, int V,
                                int nrows, void* stream) {
    LT_REQUIRE(Wq && Wd && toks && out, "lt_embed_q8_rows: null pointer");
    LT_REQUIRE(E > 0 && E % 32 == 0 && V > 0 && nrows > 0, "lt_embed_q8_rows: E=%d (multiple of 32) V=%d nrows=%d", E, V, nrows);
    int* st = device_status_ptr();
    LT_REQUIRE(st != nullptr, "lt_embed_q8_rows: status word unavailable");
    const cudaError_t e = launch_chained(k_embed_q8_rows, dim3(nrows), dim3(256), 0, (cudaStream_t)stream, Wq,
                                         (const __half*)Wd, toks, out, E, V, nrows, st);
    return check_launch("lt_embed_q8_rows", 1, e);
}

extern "C" int lt_rope_rows(float* X, int ld, const int* pos0, int nrows, int n_head, int hd, float theta,
                            void* stream) {
    LT_REQUIRE(X && pos0, "lt_rope_rows: null pointer");
    LT_REQUIRE(nrows > 0 && n_head > 0 && hd > 0 && hd % 2 == 0 && ld >= n_head * hd,
               "lt_rope_rows: nrows=%d n_head=%d hd=%d ld=%d", nrows, n_head, hd, ld);
    const long total = (long)nrows * n_head * (hd / 2);
    k_rope_rows<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>(X, ld, pos0, nrows, n_head, hd, theta);
    return check_launch("lt_rope_rows");
}

static int check_seqs(const char* what, const lt_row_seqs* S, int B, int T) {
    LT_REQUIRE(S != nullptr && B > 0 && B <= LT_ROW_SEQS && T > 0, "%s: B=%d (1 to %d) T=%d", what, B, LT_ROW_SEQS, T);
    for (int b = 0; b < B; b++) {
        LT_REQUIRE(S->k[b] && S->v[b] && S->len[b], "%s: null pointer", what);
        LT_REQUIRE(S->start[b] >= 0 && S->start[b] + (long)T <= S->max_seq[b], "%s: %d + %d positions exceed %d", what, S->start[b], T,
                   S->max_seq[b]);
        for (int o = 0; o < b; o++) LT_REQUIRE(S->len[o] != S->len[b], "%s: sequences %d and %d have one length", what, o, b);
    }
    return LT_OK;
}

extern "C" int lt_rope_append_rows(float* X, int ld, const lt_row_seqs* seqs, int B, int T, int nh, int nkv, int hd, float theta,
                                   void* stream) {
    const int rc = check_seqs("lt_rope_append_rows", seqs, B, T);
    if (rc != LT_OK) return rc;
    LT_REQUIRE(X && nh > 0 && nkv > 0 && hd > 0 && hd % 2 == 0 && ld >= (nh + 2 * nkv) * hd && (long)B * T < (1L << 31),
               "lt_rope_append_rows: nh=%d nkv=%d hd=%d ld=%d", nh, nkv, hd, ld);
    const long threads = (long)B * T * (hd / 2);
    const int heads = nh + 2 * nkv;
    const int per = threads >= 512L * sm_count() ? heads : (heads + 3) / 4;     // few rows: the heads of a row in four parts
    dim3 grid((unsigned)((threads + 255) / 256), (unsigned)((heads + per - 1) / per));
    k_rope_append_rows<<<grid, 256, 0, (cudaStream_t)stream>>>(X, ld, *seqs, B, T, nh, nkv, hd, theta, per);
    return check_launch("lt_rope_append_rows");
}

extern "C" int lt_append_kv_rows(float* kbase, const float* ksrc, float* vbase, const float* vsrc, int src_ld, int* len,
                                 int width, int max_seq, int nrows, int incr, void* stream) {
    LT_REQUIRE(kbase && ksrc && vbase && vsrc && len, "lt_append_kv_rows: null pointer");
    LT_REQUIRE(width > 0 && max_seq > 0 && nrows > 0 && src_ld >= width,
               "lt_append_kv_rows: width=%d max_seq=%d nrows=%d src_ld=%d", width, max_seq, nrows, src_ld);
    int* st = device_status_ptr();
    LT_REQUIRE(st != nullptr, "lt_append_kv_rows: status word unavailable");
    const long total = (long)nrows * width;
    int blocks = (int)((total + 255) / 256);
    if (blocks > 1184) blocks = 1184;
    k_append_kv_rows<<<blocks, 256, 0, (cudaStream_t)stream>>>(kbase, ksrc, vbase, vsrc, src_ld, len, width, max_seq,
                                                              nrows, st);
    int n = 1;
    if (incr) {
        k_add_len<<<1, 32, 0, (cudaStream_t)stream>>>(len, nrows, max_seq);
        n = 2;
    }
    return check_launch("lt_append_kv_rows", n);
}

extern "C" int lt_silu_mul_quant_rows(const float* g, const float* u, int ld, int8_t* Xq, uint16_t* Xd, int K, int rows,
                                      void* stream) {
    LT_REQUIRE(g && u && Xq && Xd, "lt_silu_mul_quant_rows: null pointer");
    LT_REQUIRE(K > 0 && K % 32 == 0 && rows > 0 && ld >= K, "lt_silu_mul_quant_rows: K=%d rows=%d ld=%d", K, rows, ld);
    const long blocks32 = (long)rows * (K / 32);
    // more than 40 blocks per SM: 5120 blocks 2.16 us, 2.21 with four elements per thread, 6144 2.46 and 2.25
    const bool quads = blocks32 > 40L * sm_count() && aligned16(g) && aligned16(u) && ld % 4 == 0 && (reinterpret_cast<uintptr_t>(Xq) & 3u) == 0;
    const cudaError_t e =
        quads ? launch_chained(k_silu_mul_quant_rows, dim3((unsigned)((blocks32 + 31) / 32)), dim3(256), 0, (cudaStream_t)stream, g, u,
                               ld, Xq, (__half*)Xd, K, rows)
              : launch_chained(k_silu_mul_quant_rows_lane, dim3((unsigned)((blocks32 + 7) / 8)), dim3(256), 0, (cudaStream_t)stream, g, u,
                               ld, Xq, (__half*)Xd, K, rows);
    return check_launch("lt_silu_mul_quant_rows", 1, e);
}

extern "C" int lt_attn_prefill(const float* Q, int q_ld, const float* K, const float* V, const int* len, float* OUT,
                               int out_ld, int hd, int nh, int nkv, float scale, int nrows, int maxt, void* stream) {
    LT_REQUIRE(Q && K && V && len && OUT, "lt_attn_prefill: null pointer");
    LT_REQUIRE(hd == 64 || hd == 128, "lt_attn_prefill: hd=%d (64 and 128 are built)", hd);
    LT_REQUIRE(nh > 0 && nkv > 0 && nh % nkv == 0, "lt_attn_prefill: nh=%d must be a positive multiple of nkv=%d", nh, nkv);
    LT_REQUIRE(nrows > 0 && maxt >= nrows && maxt <= PREFILL_MAXT, "lt_attn_prefill: nrows=%d maxt=%d (maxt in nrows..%d)", nrows, maxt, PREFILL_MAXT);
    LT_REQUIRE(q_ld >= nh * hd && out_ld >= nh * hd && q_ld % 4 == 0, "lt_attn_prefill: q_ld=%d out_ld=%d", q_ld, out_ld);
    LT_REQUIRE(out_ld % 2 == 0 && (reinterpret_cast<uintptr_t>(OUT) & 7u) == 0 && (reinterpret_cast<uintptr_t>(V) & 7u) == 0,
               "lt_attn_prefill: OUT and V must be 8-byte aligned, out_ld even");
    LT_REQUIRE(aligned16(Q) && aligned16(K), "lt_attn_prefill: Q and K must be 16-byte aligned");
    cudaStream_t s = (cudaStream_t)stream;
    if (hd == 64) return pick_attn_prefill<64>(Q, q_ld, K, V, len, OUT, out_ld, nh, nkv, scale, nrows, maxt, s);
    return pick_attn_prefill<128>(Q, q_ld, K, V, len, OUT, out_ld, nh, nkv, scale, nrows, maxt, s);
}

extern "C" int lt_attn_prefill_rows(const float* Q, int q_ld, const lt_row_seqs* seqs, int B, int T, float* OUT, int out_ld, int hd,
                                    int nh, int nkv, float scale, void* stream) {
    int rc = check_seqs("lt_attn_prefill_rows", seqs, B, T);
    if (rc != LT_OK) return rc;
    int maxt = 0;
    AttnSeqs S = {};
    bool ok = Q && OUT && (hd == 64 || hd == 128) && nh > 0 && nkv > 0 && nh % nkv == 0 && q_ld >= nh * hd && out_ld >= nh * hd &&
              q_ld % 4 == 0 && out_ld % 2 == 0 && (reinterpret_cast<uintptr_t>(OUT) & 7u) == 0 && aligned16(Q);
    for (int b = 0; b < B; b++) {
        S.k[b] = seqs->k[b];
        S.v[b] = seqs->v[b];
        S.total[b] = seqs->start[b] + T;
        if (S.total[b] > maxt) maxt = S.total[b];
        ok = ok && aligned16(S.k[b]) && (reinterpret_cast<uintptr_t>(S.v[b]) & 7u) == 0;
    }
    cudaStream_t s = (cudaStream_t)stream;
    if (ok && maxt <= PREFILL_MAXT) {
        rc = hd == 64 ? pick_attn_prefill_rows<64>(Q, q_ld, S, B, OUT, out_ld, nh, nkv, scale, T, maxt, s)
                      : pick_attn_prefill_rows<128>(Q, q_ld, S, B, OUT, out_ld, nh, nkv, scale, T, maxt, s);
        if (rc != LT_ERR_UNSUPPORTED) return rc;
    }
    for (int b = 0; b < B; b++) {      // short chunks, and what is refused: one at a time
        rc = lt_attn_prefill(Q + (long)b * T * q_ld, q_ld, S.k[b], S.v[b], seqs->len[b], OUT + (long)b * T * out_ld, out_ld, hd, nh, nkv,
                             scale, T, S.total[b], stream);
        if (rc != LT_OK) return rc;
    }
    return LT_OK;
}
