// Weight gradients of low-rank adapters: out[F, R] = alpha * X^T S for a wide activation X [N, F] and a skinny
// factor S [N, R] (R = 8, 16 or 32), both bf16, reduced over the N tokens.
//
// The reference computes these as GEMMs like any other (axis/compile.py:270-305: dA = x^T (g B^T), dB = (x A)^T g);
// with R = 16 such a product is a stream over X — 16 flops per byte — and runs at HBM speed only if X is read once,
// by many CTAs, with next to no work per byte.  A tcgen05 tile would be 1/16 full and a split-K launch per product
// costs more in fill, drain and reduction than the product itself.  So: one launch covers up to sixteen products (all
// adapters of a layer); a
// CTA takes 256 columns of one X and a slice of the tokens, stages 64-token pieces with cp.async, multiplies with
// mma.sync (the fragments are transposed on the way out of shared memory by ldmatrix.trans) and leaves an fp32
// partial [F, R] per token slice; a second small kernel sums the slices in a fixed order (bit-reproducible), scales
// and writes either [F, R] or its transpose [R, F] — the layout of the adapter's other factor.
#include <cuda_bf16.h>

#include "common.cuh"
#include "kernels.h"

static __device__ __forceinline__ uint32_t lg_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

#define LG_COLS 256          // columns of X per CTA
#define LG_TOK 64            // tokens per stage
#define LG_XS (LG_COLS * 2 + 16)   // padded row pitch of the X stage in bytes (conflict-free ldmatrix)
#define LG_THREADS 256

struct LoraGradProb {
    const bf16* X;
    const bf16* S;
    float* out;
    int F;                   // columns of X == rows of out
    int chunks;              // ceil(F / LG_COLS)
    int layout;              // 0: out is [F, R], 1: [R, F]
    long long ws_off;        // offset of this product's partials in the workspace (floats)
};
#define LG_MAX_PROBS 16
struct LoraGradArgs {
    LoraGradProb p[LG_MAX_PROBS];
    int count, N, nsplit, tok_per;
    float alpha;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N_> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N_) : "memory"); }
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x2_t(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16_16816(float* c, const uint32_t* a, const uint32_t* b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// NT = R / 8.  grid = (column chunks of all products, token slices)
template <int NT>
__global__ void __launch_bounds__(LG_THREADS) k_lora_grad_partial(const LoraGradArgs a, float* __restrict__ ws) {
    constexpr int R = NT * 8;
    constexpr int SS = R * 2 + 16;                         // padded row pitch of the S stage
    constexpr int STAGE = LG_TOK * LG_XS + LG_TOK * SS;
    extern __shared__ __align__(128) uint8_t lg_smem[];
    const uint32_t sbase = lg_smem_u32(lg_smem);
    int g = 0, chunk = blockIdx.x;
    while (g + 1 < a.count && chunk >= a.p[g].chunks) { chunk -= a.p[g].chunks; g++; }
    const LoraGradProb P = a.p[g];
    const int f0 = chunk * LG_COLS;
    const int split = blockIdx.y;
    const int t_begin = split * a.tok_per, t_end = min(a.N, t_begin + a.tok_per);
    const int nstage = t_end > t_begin ? (t_end - t_begin + LG_TOK - 1) / LG_TOK : 0;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    auto load_stage = [&](int st, int buf) {
        const int t0 = t_begin + st * LG_TOK;
        const uint32_t xs = sbase + buf * STAGE, ss = xs + LG_TOK * LG_XS;
        // X: 64 rows x 32 chunks of 16 bytes; out-of-range rows / columns are zero-filled
#pragma unroll
        for (int q = 0; q < (LG_TOK * LG_COLS / 8) / LG_THREADS; q++) {
            const int idx = q * LG_THREADS + tid;
            const int r = idx >> 5, c8 = idx & 31;
            const int t = t0 + r, f = f0 + c8 * 8;
            const bool ok = t < t_end && f < P.F;
            cp_async16(xs + r * LG_XS + c8 * 16, ok ? (const void*)(P.X + (long long)t * P.F + f) : (const void*)P.X, ok ? 16 : 0);
        }
        // S: 64 rows x NT chunks
        if (tid < LG_TOK * NT) {
            const int r = tid / NT, c8 = tid % NT;
            const int t = t0 + r;
            const bool ok = t < t_end;
            cp_async16(ss + r * SS + c8 * 16, ok ? (const void*)(P.S + (long long)t * R + c8 * 8) : (const void*)P.S, ok ? 16 : 0);
        }
        cp_async_commit();
    };

    float acc[2][NT][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[i][j][e] = 0.f;

    if (nstage > 0) load_stage(0, 0);
    for (int st = 0; st < nstage; st++) {
        if (st + 1 < nstage) { load_stage(st + 1, (st + 1) & 1); cp_async_wait<1>(); }
        else cp_async_wait<0>();
        __syncthreads();
        const uint32_t xs = sbase + (st & 1) * STAGE, ss = xs + LG_TOK * LG_XS;
        const int mi = lane >> 3, ri = lane & 7;           // ldmatrix: matrix index and row inside it
#pragma unroll
        for (int ks = 0; ks < LG_TOK / 16; ks++) {
            const int t0 = ks * 16;
            uint32_t bfr[NT][2];
#pragma unroll
            for (int nt = 0; nt < NT; nt++)                // S^T fragments: stored rows are tokens (k), columns ranks (n)
                ldsm_x2_t(ss + (t0 + (mi & 1) * 8 + ri) * SS + nt * 16, bfr[nt]);
#pragma unroll
            for (int mt = 0; mt < 2; mt++) {
                const int fc = warp * 32 + mt * 16;
                uint32_t afr[4];                            // X^T fragments: m0 (f 0-7, t 0-7) m1 (f 8-15, t 0-7) m2 (f 0-7, t 8-15) m3
                ldsm_x4_t(xs + (t0 + (mi >> 1) * 8 + ri) * LG_XS + (fc + (mi & 1) * 8) * 2, afr);
#pragma unroll
                for (int nt = 0; nt < NT; nt++) mma_bf16_16816(acc[mt][nt], afr, bfr[nt]);
            }
        }
        __syncthreads();
    }
    // partial [split][F][R]
    float* dst = ws + P.ws_off + (long long)split * P.F * R;
    const int gq = lane >> 2, q2 = (lane & 3) * 2;
#pragma unroll
    for (int mt = 0; mt < 2; mt++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int f = f0 + warp * 32 + mt * 16 + h * 8 + gq;
            if (f < P.F) {
#pragma unroll
                for (int nt = 0; nt < NT; nt++)
                    *reinterpret_cast<float2*>(dst + (long long)f * R + nt * 8 + q2) = make_float2(acc[mt][nt][h * 2], acc[mt][nt][h * 2 + 1]);
            }
        }
}

// out = alpha * sum over token slices, in slice order; layout 0: [F, R], 1: [R, F]
__global__ void k_lora_grad_reduce(const LoraGradArgs a, const float* __restrict__ ws, int R) {
    int g = blockIdx.y;
    const LoraGradProb P = a.p[g];
    const long long n = (long long)P.F * R;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float s = 0.f;
        for (int sp = 0; sp < a.nsplit; sp++) s += ws[P.ws_off + sp * n + i];
        const int f = (int)(i / R), r = (int)(i % R);
        P.out[P.layout ? (long long)r * P.F + f : i] = a.alpha * s;
    }
}

static bool g_lora_attr = false;

// X[g] [N, F[g]] bf16, S[g] [N, R] bf16 -> out[g] fp32 ([F, R], or [R, F] where layout[g] is 1).  ws: fp32 workspace of
// ws_bytes.  Returns -1 when the request is outside what the kernel serves (the caller then uses GEMMs).
int ax_lora_grad(int count, const void* const* X, const void* const* S, float* const* out, const int* F, const int* layout,
                 int N, int R, float alpha, float* ws, size_t ws_bytes, cudaStream_t st) {
    if (count < 1 || count > LG_MAX_PROBS || N < 1 || !(R == 8 || R == 16 || R == 32) || !ws) return -1;
    LoraGradArgs a = {};
    a.count = count; a.N = N; a.alpha = alpha;
    int chunks = 0, fmax = 0;
    long long fsum = 0;
    for (int g = 0; g < count; g++) {
        if (F[g] < 8 || F[g] % 8 || !aligned16(X[g]) || !aligned16(S[g]) || !out[g]) return -1;
        a.p[g].X = (const bf16*)X[g]; a.p[g].S = (const bf16*)S[g]; a.p[g].out = out[g]; a.p[g].F = F[g];
        a.p[g].layout = layout[g] ? 1 : 0;
        a.p[g].chunks = (F[g] + LG_COLS - 1) / LG_COLS;
        chunks += a.p[g].chunks; fsum += F[g]; fmax = F[g] > fmax ? F[g] : fmax;
    }
    // token slices: as many CTAs as are resident at once (three per SM) and no more — a second, partial wave would cost
    // as much as the first; at least one 64-token stage each, partials inside the workspace
    int nsplit = (3 * AX_SMS) / chunks;
    if (nsplit < 1) nsplit = 1;
    const int max_split = (N + LG_TOK - 1) / LG_TOK;
    if (nsplit > max_split) nsplit = max_split;
    if (nsplit > 64) nsplit = 64;
    while (nsplit > 1 && (size_t)nsplit * fsum * R * 4 > ws_bytes) nsplit--;
    if ((size_t)nsplit * fsum * R * 4 > ws_bytes) return -1;
    a.tok_per = ((N + nsplit - 1) / nsplit + LG_TOK - 1) / LG_TOK * LG_TOK;
    nsplit = (N + a.tok_per - 1) / a.tok_per;
    a.nsplit = nsplit;
    long long off = 0;
    for (int g = 0; g < count; g++) { a.p[g].ws_off = off; off += (long long)nsplit * F[g] * R; }
    const int NT = R / 8;
    const size_t smem = 2 * (size_t)(LG_TOK * LG_XS + LG_TOK * (R * 2 + 16));
    if (!g_lora_attr) {
        cudaFuncSetAttribute(k_lora_grad_partial<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * (LG_TOK * LG_XS + LG_TOK * 32));
        cudaFuncSetAttribute(k_lora_grad_partial<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * (LG_TOK * LG_XS + LG_TOK * 48));
        cudaFuncSetAttribute(k_lora_grad_partial<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * (LG_TOK * LG_XS + LG_TOK * 80));
        g_lora_attr = true;
    }
    const dim3 grid(chunks, nsplit);
    if (NT == 1) k_lora_grad_partial<1><<<grid, LG_THREADS, smem, st>>>(a, ws);
    else if (NT == 2) k_lora_grad_partial<2><<<grid, LG_THREADS, smem, st>>>(a, ws);
    else k_lora_grad_partial<4><<<grid, LG_THREADS, smem, st>>>(a, ws);
    const int rb = (int)(((long long)fmax * R + 255) / 256);
    k_lora_grad_reduce<<<dim3(rb > 592 ? 592 : rb, count), 256, 0, st>>>(a, ws, R);
    return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

// ── the skinny products of an adapter: out[N, R] = alpha * X W (W [F, R]) or alpha * X W^T (W [R, F]) ──────────────────
// u = x A in the forward and t = g B^T in the backward: again a stream over the wide operand with 16 flops per byte.
// A CTA takes TOK tokens and walks F in pieces of COLS columns; its eight warps are the row tiles times equal shares of a
// piece's depth, and the partial accumulators of a row tile meet in shared memory.  What bounds it is what an SM takes in:
// besides its X a CTA reads all of W, from L2: at 32 tokens a CTA half as many bytes as X at rank 16, as many at rank 32.  Hence 64 tokens, and products of one X (the adapters of q, k and v, of gate and up) as M members
// of one CTA, where X is staged once for all of them; one barrier a piece, all stages in flight from the start, and
// neighbouring token blocks begin at different pieces, or all SMs ask for the same lines of W at the same time.
// Rank 16, three products of one X, 8192 x 1536: 25.4 us with 32 tokens and a CTA per product, 17.0 with 64 and members,
// 15.5 with the pieces turned, 15.1 with all stages in flight; one product of 8192 x 4096 24.0 -> 16.4; two of their own
// 8192 x 4096 39.6 -> 25.0 (5.4 TB/s).

struct LoraProjProb {
    const bf16* X;
    const bf16* W;
    bf16* out;
    int F;
};
struct LoraProjArgs {
    LoraProjProb p[3];
    int count, N, S;         // S: CTAs of a cluster that share out the depth of a token block
    float alpha;
};

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x2(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
}

// TB = 0: W is [F, R]; TB = 1: W is [R, F].
// grid = (token blocks * S, products); M > 1: one row of blocks for M products of the same X and F.
// TOK 64 with pieces of 128 columns (64 where the members' W would leave one CTA to an SM), or 32 with pieces of 256.
template <int NT, int TB, int M, int TOK> struct LoraProj {
    static constexpr int R = NT * 8, COLS = TOK == 32 ? 256 : (R * M > 64 ? 64 : 128);
    static constexpr int XS = COLS * 2 + 16, WS = TB ? XS : (R == 8 ? 16 : R * 2 + 16), WROWS = TB ? R : COLS;    // padded pitches: conflict-free ldmatrix
    static constexpr int XBYTES = TOK * XS, WBYTES = WROWS * WS, STAGE = XBYTES + M * WBYTES;
    static constexpr int ROOM = 113 * 1024;                // two CTAs to an SM
    static constexpr int STAGES = STAGE * 4 <= ROOM ? 4 : 3;
    static constexpr int RT = TOK / 16, KQ = 8 / RT;       // row tiles, shares of a piece's depth: one warp each
    static constexpr int RP = M * R % 16 ? M * R : M * R + 8;              // row pitch of the sums in floats: rows of a fragment in banks of their own
    static constexpr int RED = (KQ + 1) * TOK * RP * 4; // the shares and their sum
    static constexpr int SMEM = STAGES * STAGE > RED ? STAGES * STAGE : RED;
    static_assert(SMEM <= ROOM, "two CTAs to an SM");
};
template <int NT, int TB, int M, int TOK>
__global__ void __launch_bounds__(256) k_lora_proj(const __grid_constant__ LoraProjArgs a) {
    using L = LoraProj<NT, TB, M, TOK>;
    constexpr int R = L::R, COLS = L::COLS, XS = L::XS, WS = L::WS, XBYTES = L::XBYTES, WBYTES = L::WBYTES, STAGE = L::STAGE, STAGES = L::STAGES, RM = R * M, RP = L::RP;
    extern __shared__ __align__(128) uint8_t lg_smem[];
    const uint32_t sbase = lg_smem_u32(lg_smem);
    const int g0 = blockIdx.y;                             // 0 where M > 1
    const bf16* const X = a.p[g0].X;
    const int F = a.p[g0].F;
    const int part = blockIdx.x % a.S, t0 = blockIdx.x / a.S * TOK;     // a.S CTAs along x are one cluster
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int pieces = (F + COLS - 1) / COLS;
    const int st0 = (int)((long long)pieces * part / a.S), nstage = (int)((long long)pieces * (part + 1) / a.S) - st0;
    int at = nstage > 0 ? st0 + (int)(blockIdx.x / a.S) % nstage : 0;       // the piece to load next: neighbours start apart
    pdl_enter();

    auto load_stage = [&](int st) {
        const int f0 = at * COLS;
        at = at + 1 == st0 + nstage ? st0 : at + 1;
        const uint32_t xs = sbase + (st % STAGES) * STAGE;
#pragma unroll
        for (int q = 0; q < TOK * (COLS / 8) / 256; q++) {           // X: 64 rows of COLS / 8 chunks
            const int idx = q * 256 + tid;
            const int r = idx / (COLS / 8), c8 = idx % (COLS / 8);
            const int t = t0 + r, f = f0 + c8 * 8;
            const bool ok = t < a.N && f < F;
            cp_async16(xs + r * XS + c8 * 16, ok ? (const void*)(X + (long long)t * F + f) : (const void*)X, ok ? 16 : 0);
        }
#pragma unroll
        for (int m = 0; m < M; m++) {
            const bf16* const W = a.p[M > 1 ? m : g0].W;
            const uint32_t ws_ = xs + XBYTES + m * WBYTES;
#pragma unroll
            for (int q = 0; q < (R * COLS / 8 + 255) / 256; q++) {      // W: R * COLS / 8 chunks either way
                const int idx = q * 256 + tid;
                if (R * COLS / 8 % 256 && idx >= R * COLS / 8) break;
                const int r = TB ? idx / (COLS / 8) : idx / NT, c8 = TB ? idx % (COLS / 8) : idx % NT;
                const int f = TB ? f0 + c8 * 8 : f0 + r;
                const bool ok = f < F;
                cp_async16(ws_ + r * WS + c8 * 16, ok ? (const void*)(W + (TB ? (long long)r * F + f : (long long)f * R + c8 * 8)) : (const void*)W, ok ? 16 : 0);
            }
        }
    };

    float acc[M * NT][4];
#pragma unroll
    for (int j = 0; j < M * NT; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[j][e] = 0.f;
    const int mt = warp % L::RT, kq = warp / L::RT;        // row tile, share of the piece's depth
    const int mi = lane >> 3, ri = lane & 7;

#pragma unroll
    for (int st = 0; st < STAGES; st++) { if (st < nstage) load_stage(st); cp_async_commit(); }
    for (int st = 0; st < nstage; st++) {
        if (st == 0) cp_async_wait<STAGES - 1>(); else cp_async_wait<STAGES - 2>();
        __syncthreads();                                    // piece st is there, and everyone has left piece st - 1
        if (st) { if (st - 1 + STAGES < nstage) load_stage(st - 1 + STAGES); cp_async_commit(); }
        const uint32_t xs = sbase + (st % STAGES) * STAGE;
#pragma unroll
        for (int ks = 0; ks < COLS / L::KQ / 16; ks++) {
            const int k0 = kq * (COLS / L::KQ) + ks * 16;
            uint32_t afr[4];                                 // X fragments: (rows 0-7, k 0-7) (rows 8-15, k 0-7) (rows 0-7, k 8-15) (rows 8-15, k 8-15)
            ldsm_x4(xs + (mt * 16 + (mi & 1) * 8 + ri) * XS + (k0 + (mi >> 1) * 8) * 2, afr);
#pragma unroll
            for (int m = 0; m < M; m++) {
                const uint32_t ws_ = xs + XBYTES + m * WBYTES;
#pragma unroll
                for (int nt = 0; nt < NT; nt += 2) {         // W^T stored [n][k], or W stored [k][n]; two column tiles a load
                    uint32_t bfr[4];
                    const int n8 = nt + (NT > 1 ? mi >> 1 : 0);
                    const uint32_t at = TB ? ws_ + (n8 * 8 + ri) * WS + (k0 + (mi & 1) * 8) * 2 : ws_ + (k0 + (mi & 1) * 8 + ri) * WS + n8 * 16;
                    if (NT == 1) { if (TB) ldsm_x2(at, bfr); else ldsm_x2_t(at, bfr); }
                    else { if (TB) ldsm_x4(at, bfr); else ldsm_x4_t(at, bfr); }
                    mma_bf16_16816(acc[m * NT + nt], afr, bfr);
                    if (NT > 1) mma_bf16_16816(acc[m * NT + (nt + 1) % NT], afr, bfr + 2);
                }
            }
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    // the depth shares of a row tile meet in shared memory (the operand stages are free now)
    float* red = reinterpret_cast<float*>(lg_smem);         // [kq][TOK rows][M * R]
    const int gq = lane >> 2, q2 = (lane & 3) * 2;
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int nt = 0; nt < M * NT; nt++)
            *reinterpret_cast<float2*>(red + (kq * TOK + mt * 16 + h * 8 + gq) * RP + nt * 8 + q2) = make_float2(acc[nt][h * 2], acc[nt][h * 2 + 1]);
    __syncthreads();
    auto shares = [&](int j) {
        const int i = j / RM * RP + j % RM;
        float2 u = *reinterpret_cast<const float2*>(red + i);
#pragma unroll
        for (int q = 1; q < L::KQ; q++) {
            const float2 v = *reinterpret_cast<const float2*>(red + q * TOK * RP + i);
            u.x += v.x; u.y += v.y;
        }
        return u;
    };
    auto store = [&](int i, float2 s) {
        const int r = i / RM, m = i % RM / R, c = i % R;
        if (t0 + r < a.N) *reinterpret_cast<__nv_bfloat162*>(a.p[M > 1 ? m : g0].out + (long long)(t0 + r) * R + c) = __floats2bfloat162_rn(a.alpha * s.x, a.alpha * s.y);
    };
    if (a.S == 1) {
        for (int i = tid * 2; i < TOK * RM; i += 512) store(i, shares(i));
        return;
    }
    // the cluster's parts: every CTA leaves its sum, then finishes 1 / S of the rows from all CTAs' sums, in part order
    float* mine = red + L::KQ * TOK * RP;
    for (int i = tid * 2; i < TOK * RM; i += 512) *reinterpret_cast<float2*>(mine + i) = shares(i);
    cluster_sync();
    const int share = TOK / a.S * RM;
    for (int i = part * share + tid * 2; i < (part + 1) * share; i += 512) {
        float2 s = make_float2(0.f, 0.f);
        const uint32_t at = lg_smem_u32(mine + i);
        for (int p = 0; p < a.S; p++) {
            float2 v;
            asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %2, %3;\n\tld.shared::cluster.v2.f32 {%0, %1}, [ra];\n\t}"
                         : "=f"(v.x), "=f"(v.y) : "r"(at), "r"(p) : "memory");
            s.x += v.x; s.y += v.y;
        }
        store(i, s);
    }
    cluster_sync();   // peers have read
}

// How a launch of `count` products of N tokens, F columns (the narrowest) and rank R is cut: products as members of one CTA, tokens of a CTA, CTAs that share a CTA's walk.
struct LoraProjCut { int members, tokens, S; };
static LoraProjCut lora_proj_cut(int count, bool one_x, int N, int F, int R) {
    // Members of one X pay where a CTA per product would go beyond a resident wave (three products of rank 32, 8192 x 1536: 18.6 us as members, 24.3 each),
    // or where token blocks alone occupy the SMs, the walk is long and the member loop short (rank 16, three of 2048 x 4096 10.5 and 15.0 us, two of 3000 x 2048 7.9 and 9.1;
    // rank 32, three of 3000 x 1536 11.3 and 9.4; two of 256 x 1024 3.8 and 3.4; rank 16, three of 4999 x 776 8.5 and 6.7, of 2006 x 864 7.9 and 5.6).
    const int blocks = (N + 63) / 64;
    LoraProjCut c = {one_x && ((blocks >= 32 && R * count <= 64 && F >= 1536) || blocks * count > 2 * AX_SMS) ? count : 1, 64, 1};
    const int rows = c.members > 1 ? 1 : count;
    // Depth split: a CTA that walks all of F alone is a chain of round trips, and few token blocks leave SMs idle.  Never beyond one resident wave, two CTAs an SM, which is 148
    // clusters of two, 72 of four or 32 of eight: x A of 8192 x 1536 in blocks of 32 tokens 11.0 us on 256 CTAs, 13.9 us on 512; 74 clusters of four, 4707 x 6376 rank 32,
    // 35.8 us, 24.9 in two; 34 of eight, 538 x 2320 rank 8, 6.8, 4.4 in four.  The barriers and the sum take 1 us, what some 500 columns do, one CTA / two: rank 8, 6510 x 232
    // 2.1 / 3.4, 9458 x 160 2.4 / 3.8; rank 16, 5241 x 320 3.1 / 4.4, 3196 x 712 4.1 / 4.6; 1936 columns 10.7 / 8.9.
    auto fits = [](long long n, int S) { return n <= (S == 2 ? AX_SMS : S == 4 ? 72 : 32); };
    while (c.S < 8 && fits((long long)blocks * rows, 2 * c.S) && F >= 1024 && F * c.members >= 1024 * c.S) c.S *= 2;
    // Where even the split leaves SMs without a CTA the walk's length counts, not W's traffic: 32 tokens and pieces of 256 columns.
    // Rank 16, one product: 70 x 4096 4.4 us in blocks of 64, 3.5 of 32; 1024 x 4096 6.3 and 5.2, 4160 x 416 3.8 and 3.1; above, 2048 x 4096 7.3 and 8.1.
    if (c.members == 1 && blocks * rows * c.S <= AX_SMS) {
        const int small = (N + 31) / 32;
        c.tokens = 32;
        c.S = 1;
        while (c.S < 8 && fits((long long)small * rows, 2 * c.S) && F >= (c.S == 1 ? 768 : 512 * c.S)) c.S *= 2;
    }
    return c;
}
int ax_lora_proj_cut(int count, int one_x, int N, int F, int R) {
    const LoraProjCut c = lora_proj_cut(count, one_x != 0, N, F, R);
    return c.members << 16 | c.tokens << 8 | c.S;
}

template <int NT, int TB, int M, int TOK> static int lora_proj_launch(const LoraProjArgs& a, int S, cudaStream_t st) {
    using L = LoraProj<NT, TB, M, TOK>;
    static const cudaError_t attr = cudaFuncSetAttribute(k_lora_proj<NT, TB, M, TOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM);
    if (attr != cudaSuccess) return 3;
    LoraProjArgs b = a;
    b.S = S;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((a.N + TOK - 1) / TOK * S, M > 1 ? 1 : a.count); cfg.blockDim = dim3(256); cfg.dynamicSmemBytes = L::SMEM; cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = ax_gemm_pdl() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, k_lora_proj<NT, TB, M, TOK>, b) == cudaSuccess ? 0 : 3;
}

// out[g] [N, R] bf16 = alpha * X[g] [N, F[g]] W[g]; tb 0: W [F, R], tb 1: W [R, F].  -1 when not served.
int ax_lora_proj(int count, int tb, const void* const* X, const void* const* W, void* const* out, const int* F, int N, int R,
                 float alpha, cudaStream_t st) {
    if (count < 1 || count > 3 || N < 1 || !(R == 8 || R == 16 || R == 32) || tb < 0 || tb > 1) return -1;
    LoraProjArgs a = {};
    a.count = count; a.N = N; a.alpha = alpha;
    for (int g = 0; g < count; g++) {
        if (F[g] < 8 || F[g] % 8 || !aligned16(X[g]) || !aligned16(W[g]) || !out[g] || ((uintptr_t)out[g] & 3)) return -1;
        a.p[g].X = (const bf16*)X[g]; a.p[g].W = (const bf16*)W[g]; a.p[g].out = (bf16*)out[g]; a.p[g].F = F[g];
    }
    bool one_x = true;
    int least = F[0];
    for (int g = 1; g < count; g++) { one_x = one_x && X[g] == X[0] && F[g] == F[0]; least = F[g] < least ? F[g] : least; }
    const LoraProjCut c = lora_proj_cut(count, one_x, N, least, R);
#define LPM(NT_, TB_) (c.members == 3 ? lora_proj_launch<NT_, TB_, 3, 64>(a, c.S, st) : c.members == 2 ? lora_proj_launch<NT_, TB_, 2, 64>(a, c.S, st) \
                       : c.tokens == 64 ? lora_proj_launch<NT_, TB_, 1, 64>(a, c.S, st) : lora_proj_launch<NT_, TB_, 1, 32>(a, c.S, st))
#define LP(NT_) (tb ? LPM(NT_, 1) : LPM(NT_, 0))
    return R == 8 ? LP(1) : (R == 16 ? LP(2) : LP(4));
#undef LP
#undef LPM
}
