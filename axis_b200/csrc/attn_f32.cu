// Causal grouped-query attention in exact fp32 for head dims from 12 to 64 (rows in whole 16-byte pieces): the parity mode at its usual sizes.
// attn_simt.cu serves everything else, and what is faster there (see ax_attn_f32_ctas).
//
// Bound by shared-memory reads and latency there: a lane of attn_simt.cu owns one row of the walked tile, and 16 FMAs take one read of its own row and four
// broadcasts, eight cycles of the shared-memory pipe for four of the FMA pipes.  Here a warp owns 16 rows and a lane 4 x 4 of its 16 x 32 scores (rows rg + 4 i, columns
// kg + 8 j; rg = lane / 8, kg = lane % 8), so that eight reads that each fall in different banks feed 64 FMAs, and the second product (P V, dS K, P^T dO, dS^T Q) has
// four rows and DH / 8 columns to a lane, with the probabilities going through shared memory as [column][16 rows].  A block is four warps, 64 rows; tiles of
// 32 rows of the walked operands are double-buffered by cp.async, and where blocks are few a cluster takes the tiles in turn (see attn_simt.cu).  No atomics, sums in a
// fixed order.  B2 H8 KV4 T256 DH32, us in attn_simt.cu / here, forward and backward with the row
// dots: 14.9 and 42.2 / 12.3 and 30.4; B2 H12 KV4 T900 DH64 215 and 633 / 127 and 431.  2-norm errors against float64 (T 128 to 900) are 0.79 to 1.01 times those there.
#include <math.h>

#include <initializer_list>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

#define FW 4             // warps per block
#define FTH (FW * 32)
#define FB (FW * 16)     // rows per block
#define FT 32            // rows of a walked tile

template <int DHP> struct F32Att {
    static constexpr int LD = DHP + 4, NC = DHP / 8, TILE = FT * LD, OWN = FB * LD, P = FT * 16;     // floats; LD: rows kg, kg + 1, ... in different banks
};
// ROWS rows of `stride` floats from r0 of a [T, DH] window; rows past T are zeros, columns past DH stay what they were (their sums are never stored)
template <int DHP, int ROWS>
__device__ __forceinline__ void fa_load(float* dst, const float* src, long long stride, int r0, int T, int DH) {
    constexpr int Q = DHP / 4;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(dst);
#pragma unroll
    for (int i = 0; i < ROWS * Q / FTH; i++) {
        const int e = threadIdx.x + i * FTH, r = e / Q, d = e % Q * 4;
        const bool in = r0 + r < T;
        const float* p = in ? src + (long long)(r0 + r) * stride + d : src;
        if (d < DH) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + (r * F32Att<DHP>::LD + d) * 4), "l"(p), "r"(in ? 16 : 0) : "memory");
    }
}
__device__ __forceinline__ void fa_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void fa_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
// out[i][j] = <row i of this lane, column j of this lane>; a and b point at the first of either
template <int DHP> __device__ __forceinline__ void fa_dot(const float* a, const float* b, int DH, float (&out)[4][4]) {
    constexpr int LD = F32Att<DHP>::LD;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) out[i][j] = 0.f;
#pragma unroll 4
    for (int d = 0; d < DH; d += 4) {
        float4 x[4], y[4];
#pragma unroll
        for (int i = 0; i < 4; i++) { x[i] = *reinterpret_cast<const float4*>(a + i * 4 * LD + d); y[i] = *reinterpret_cast<const float4*>(b + i * 8 * LD + d); }
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                out[i][j] = fmaf(x[i].x, y[j].x, out[i][j]); out[i][j] = fmaf(x[i].y, y[j].y, out[i][j]);
                out[i][j] = fmaf(x[i].z, y[j].z, out[i][j]); out[i][j] = fmaf(x[i].w, y[j].w, out[i][j]);
            }
    }
}
// p[i][j] -> the warp's [column][16 rows], place rg * 4 + i for row rg + 4 i
__device__ __forceinline__ void fa_put(float* P, const float (&p)[4][4], int rg, int kg) {
#pragma unroll
    for (int j = 0; j < 4; j++) *reinterpret_cast<float4*>(P + (kg + 8 * j) * 16 + rg * 4) = make_float4(p[0][j], p[1][j], p[2][j], p[3][j]);
}
// acc[i][c] += p[column][row i] * tile[column][c] over the 32 columns; c: kg * 4 .. + 3 and 32 further on
template <int DHP> __device__ __forceinline__ void fa_axpy(float (&acc)[4][DHP / 8], const float* P, const float* tile, int rg, int kg) {
    constexpr int LD = F32Att<DHP>::LD;
#pragma unroll 4
    for (int k = 0; k < FT; k++) {
        const float4 p = *reinterpret_cast<const float4*>(P + k * 16 + rg * 4);
#pragma unroll
        for (int c = 0; c < DHP / 32; c++) {
            const float4 v = *reinterpret_cast<const float4*>(tile + k * LD + c * 32 + kg * 4);
            const float pr[4] = {p.x, p.y, p.z, p.w}, vc[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[i][c * 4 + e] = fmaf(pr[i], vc[e], acc[i][c * 4 + e]);
        }
    }
}
template <int NC> __device__ __forceinline__ void fa_zero(float (&acc)[4][NC]) {
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int c = 0; c < NC; c++) acc[i][c] = 0.f;
}
// the columns of this lane, times f, to a row of DH
template <int NC> __device__ __forceinline__ void fa_store(float* row, const float* a, float f, int kg, int DH) {
#pragma unroll
    for (int c = 0; c < NC; c += 4)
        if (c * 8 + kg * 4 < DH) *reinterpret_cast<float4*>(row + c * 8 + kg * 4) = make_float4(a[c] * f, a[c + 1] * f, a[c + 2] * f, a[c + 3] * f);
}
// What a cluster merges lies in shared memory as [piece][thread] of float4.  The pieces at `at` of all S ranks, added in rank order (SUM of a stored one: times w[rank]).  All S
// reads are under way before the first is used: where each waited for the one before it, a merge took 6 us (dK / dV of B5 H12 KV12 T13 DH16 over two CTAs: 12.0 us,
// 6.2 with one CTA and no merge).
__device__ __forceinline__ float4 fa_peer4(const float4* p, int rank) {
    float4 x;
    asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [ra];\n\t}"
                 : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank) : "memory");
    return x;
}
template <int S, int N> __device__ __forceinline__ void fa_gather(const float4* at, const float* w, float* a) {
#pragma unroll
    for (int c = 0; c < N; c += 4) {
        float4 x[S];
#pragma unroll
        for (int z = 0; z < S; z++) x[z] = fa_peer4(at + c / 4 * FTH, z);
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int z = 0; z < S; z++) {
            const float f = w ? w[z] : 1.f;
            t.x = fmaf(x[z].x, f, t.x); t.y = fmaf(x[z].y, f, t.y); t.z = fmaf(x[z].z, f, t.z); t.w = fmaf(x[z].w, f, t.w);
        }
        a[c] = t.x; a[c + 1] = t.y; a[c + 2] = t.z; a[c + 3] = t.w;
    }
}
// rows of this lane's four (N columns each, from piece 0 of a) -> pieces
template <int N> __device__ __forceinline__ void fa_leave(float4* x, const float (&a)[4][N]) {
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int c = 0; c < N; c += 4) x[(i * N + c) / 4 * FTH] = make_float4(a[i][c], a[i][c + 1], a[i][c + 2], a[i][c + 3]);
}
// f(integral constant S) for the sizes of a cluster
template <typename F> __device__ __forceinline__ void fa_of_size(int S, F f) {
    if (S == 2) f(std::integral_constant<int, 2>());
    else if (S == 4) f(std::integral_constant<int, 4>());
    else f(std::integral_constant<int, 8>());
}
// over the eight lanes of a row
__device__ __forceinline__ float fa_max8(float x) {
#pragma unroll
    for (int o = 1; o < 8; o *= 2) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}
__device__ __forceinline__ float fa_sum8(float x) {
#pragma unroll
    for (int o = 1; o < 8; o *= 2) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

template <int DHP, bool SHARE>
__global__ void __launch_bounds__(FTH)
k_attn_fwd_f32(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v, float* __restrict__ o, float* __restrict__ lse, AttnShape s, int ctas) {
    using F = F32Att<DHP>;
    extern __shared__ __align__(16) float smem[];
    float* Qs = smem;
    float* Ks = Qs + F::OWN;             // two tiles each
    float* Vs = Ks + 2 * F::TILE;
    const int b = blockIdx.z, h = blockIdx.y, g = h / (s.H / s.KV), warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rg = lane >> 3, kg = lane & 7;
    float* P = Vs + 2 * F::TILE + warp * F::P;
    const int S = SHARE ? ctas : 1, part = SHARE ? blockIdx.x % S : 0, r0 = (gridDim.x / S - 1 - blockIdx.x / S) * FB, t0 = r0 + warp * 16;       // the longest rows first
    const float* kb = k + b * s.kb + g * s.kh;
    const float* vb = v + b * s.kb + g * s.kh;
    const int ntiles = min(r0 + FB - 1, s.T - 1) / FT + 1;
    pdl_enter();
    fa_load<DHP, FB>(Qs, q + b * s.qb + h * s.qh, s.qt, r0, s.T, s.DH);
    if (part < ntiles) {
        fa_load<DHP, FT>(Ks, kb, s.kt, part * FT, s.T, s.DH);
        fa_load<DHP, FT>(Vs, vb, s.kt, part * FT, s.T, s.DH);
    }
    fa_commit();
    float m[4], l[4], acc[4][F::NC];     // l: this lane's share of the row sum
#pragma unroll
    for (int i = 0; i < 4; i++) { m[i] = -3.0e38f; l[i] = 0.f; }
    fa_zero(acc);
    for (int kt = part, it = 0; kt < ntiles; kt += S, it++) {
        fa_wait();
        __syncthreads();
        const int cur = it & 1;
        if (kt + S < ntiles) {
            fa_load<DHP, FT>(Ks + (cur ^ 1) * F::TILE, kb, s.kt, (kt + S) * FT, s.T, s.DH);
            fa_load<DHP, FT>(Vs + (cur ^ 1) * F::TILE, vb, s.kt, (kt + S) * FT, s.T, s.DH);
        }
        fa_commit();
        if (kt * FT > t0 + 15) continue;
        float sc[4][4];
        fa_dot<DHP>(Qs + (warp * 16 + rg) * F::LD, Ks + cur * F::TILE + kg * F::LD, s.DH, sc);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int last = t0 + rg + 4 * i - kt * FT - kg;                  // 8 j of the row's own key
            float mx = -3.0e38f;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                sc[i][j] = 8 * j <= last ? sc[i][j] * s.scale : -3.0e38f;
                mx = fmaxf(mx, sc[i][j]);
            }
            const float mn = fmaxf(m[i], fa_max8(mx)), corr = expf(m[i] - mn);
            l[i] *= corr;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                sc[i][j] = 8 * j <= last ? expf(sc[i][j] - mn) : 0.f;
                l[i] += sc[i][j];
            }
            m[i] = mn;
#pragma unroll
            for (int c = 0; c < F::NC; c++) acc[i][c] *= corr;
        }
        fa_put(P, sc, rg, kg);
        __syncwarp();
        fa_axpy<DHP>(acc, P, Vs + cur * F::TILE, rg, kg);
        __syncwarp();
    }
    if (SHARE) {                         // merge: sums at the largest of the ranks' maxima
        fa_wait();
        __syncthreads();
        float4* x = reinterpret_cast<float4*>(smem) + threadIdx.x;       // [row: maximum and sum; columns]
        float4* y = x + 4 * FTH;
#pragma unroll
        for (int i = 0; i < 4; i++) x[i * FTH] = make_float4(m[i], l[i], 0.f, 0.f);
        fa_leave<F::NC>(y, acc);
        cluster_sync();
        fa_of_size(S, [&](auto size) {
            constexpr int SS = decltype(size)::value;
            for (int i = part * 4 / SS; i < (part + 1) * 4 / SS; i++) {
                float4 ml[SS];
                float mx = -3.0e38f, ls = 0.f, w[SS], a[F::NC];
#pragma unroll
                for (int z = 0; z < SS; z++) ml[z] = fa_peer4(x + i * FTH, z);
#pragma unroll
                for (int z = 0; z < SS; z++) mx = fmaxf(mx, ml[z].x);
#pragma unroll
                for (int z = 0; z < SS; z++) { w[z] = expf(ml[z].x - mx); ls += ml[z].y * w[z]; }
                fa_gather<SS, F::NC>(y + i * (F::NC / 4) * FTH, w, a);
                ls = fa_sum8(ls);
                const int t = t0 + rg + 4 * i;
                if (t >= s.T) continue;
                fa_store<F::NC>(o + b * s.qb + h * s.qh + (long long)t * s.qt, a, 1.f / ls, kg, s.DH);
                if (lse && kg == 0) lse[((long long)b * s.H + h) * s.T + t] = mx + logf(ls);
            }
        });
        cluster_sync();                  // peers have read
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = t0 + rg + 4 * i;
        const float ls = fa_sum8(l[i]);
        if (t >= s.T) continue;
        fa_store<F::NC>(o + b * s.qb + h * s.qh + (long long)t * s.qt, acc[i], 1.f / ls, kg, s.DH);
        if (lse && kg == 0) lse[((long long)b * s.H + h) * s.T + t] = m[i] + logf(ls);
    }
}

// dQ: a warp owns 16 query rows and walks the keys.
template <int DHP, bool SHARE>
__global__ void __launch_bounds__(FTH)
k_attn_dq_f32(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v, const float* __restrict__ dO, const float* __restrict__ lse,
              const float* __restrict__ Dv, float* __restrict__ dq, AttnShape s, int ctas) {
    using F = F32Att<DHP>;
    extern __shared__ __align__(16) float smem[];
    float* Qs = smem;
    float* Gs = Qs + F::OWN;             // dO rows
    float* Ks = Gs + F::OWN;
    float* Vs = Ks + 2 * F::TILE;
    const int b = blockIdx.z, h = blockIdx.y, g = h / (s.H / s.KV), warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rg = lane >> 3, kg = lane & 7;
    float* P = Vs + 2 * F::TILE + warp * F::P;
    const int S = SHARE ? ctas : 1, part = SHARE ? blockIdx.x % S : 0, r0 = (gridDim.x / S - 1 - blockIdx.x / S) * FB, t0 = r0 + warp * 16;
    const float* kb = k + b * s.kb + g * s.kh;
    const float* vb = v + b * s.kb + g * s.kh;
    const int ntiles = min(r0 + FB - 1, s.T - 1) / FT + 1;
    pdl_enter();
    fa_load<DHP, FB>(Qs, q + b * s.qb + h * s.qh, s.qt, r0, s.T, s.DH);
    fa_load<DHP, FB>(Gs, dO + b * s.qb + h * s.qh, s.qt, r0, s.T, s.DH);
    if (part < ntiles) {
        fa_load<DHP, FT>(Ks, kb, s.kt, part * FT, s.T, s.DH);
        fa_load<DHP, FT>(Vs, vb, s.kt, part * FT, s.T, s.DH);
    }
    fa_commit();
    float L[4], D[4], acc[4][F::NC];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = t0 + rg + 4 * i;
        L[i] = t < s.T ? lse[((long long)b * s.H + h) * s.T + t] : 0.f;
        D[i] = t < s.T ? Dv[b * s.db + h * s.dh_ + (long long)t * s.dtk] : 0.f;
    }
    fa_zero(acc);
    for (int kt = part, it = 0; kt < ntiles; kt += S, it++) {
        fa_wait();
        __syncthreads();
        const int cur = it & 1;
        if (kt + S < ntiles) {
            fa_load<DHP, FT>(Ks + (cur ^ 1) * F::TILE, kb, s.kt, (kt + S) * FT, s.T, s.DH);
            fa_load<DHP, FT>(Vs + (cur ^ 1) * F::TILE, vb, s.kt, (kt + S) * FT, s.T, s.DH);
        }
        fa_commit();
        if (kt * FT > t0 + 15) continue;
        float sc[4][4], dp[4][4];
        fa_dot<DHP>(Qs + (warp * 16 + rg) * F::LD, Ks + cur * F::TILE + kg * F::LD, s.DH, sc);
        fa_dot<DHP>(Gs + (warp * 16 + rg) * F::LD, Vs + cur * F::TILE + kg * F::LD, s.DH, dp);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int t = t0 + rg + 4 * i, last = t - kt * FT - kg;
#pragma unroll
            for (int j = 0; j < 4; j++) sc[i][j] = 8 * j <= last && t < s.T ? expf(sc[i][j] * s.scale - L[i]) * (dp[i][j] - D[i]) * s.scale : 0.f;
        }
        fa_put(P, sc, rg, kg);
        __syncwarp();
        fa_axpy<DHP>(acc, P, Ks + cur * F::TILE, rg, kg);
        __syncwarp();
    }
    float* out = dq + b * s.qb + h * s.qh;
    if (SHARE) {
        fa_wait();
        __syncthreads();
        float4* x = reinterpret_cast<float4*>(smem) + threadIdx.x;
        fa_leave<F::NC>(x, acc);
        cluster_sync();
        fa_of_size(S, [&](auto size) {
            constexpr int SS = decltype(size)::value;
            for (int i = part * 4 / SS; i < (part + 1) * 4 / SS; i++) {
                float a[F::NC];
                fa_gather<SS, F::NC>(x + i * (F::NC / 4) * FTH, nullptr, a);
                const int t = t0 + rg + 4 * i;
                if (t < s.T) fa_store<F::NC>(out + (long long)t * s.qt, a, 1.f, kg, s.DH);
            }
        });
        cluster_sync();                  // peers have read
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = t0 + rg + 4 * i;
        if (t < s.T) fa_store<F::NC>(out + (long long)t * s.qt, acc[i], 1.f, kg, s.DH);
    }
}

// dK, dV: a warp owns 16 key rows of a kv head and walks the group's query heads and their causal query tiles (the sum over the group).
template <int DHP, bool SHARE>
__global__ void __launch_bounds__(FTH)
k_attn_dkv_f32(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v, const float* __restrict__ dO, const float* __restrict__ lse,
               const float* __restrict__ Dv, float* __restrict__ dk, float* __restrict__ dv, AttnShape s, int ctas) {
    using F = F32Att<DHP>;
    extern __shared__ __align__(16) float smem[];
    float* Kr = smem;
    float* Vr = Kr + F::OWN;
    float* Qs = Vr + F::OWN;
    float* Gs = Qs + 2 * F::TILE;
    const int b = blockIdx.z, g = blockIdx.y, rep = s.H / s.KV, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rg = lane >> 3, kg = lane & 7;
    float* P = Gs + 2 * F::TILE + warp * F::P;
    const int S = SHARE ? ctas : 1, part = SHARE ? blockIdx.x % S : 0, r0 = blockIdx.x / S * FB, j0 = r0 + warp * 16;       // the first key rows meet the most queries
    const int qt0 = r0 / FT, nq = (s.T + FT - 1) / FT - qt0, n_it = rep * nq;
    pdl_enter();
    fa_load<DHP, FB>(Kr, k + b * s.kb + g * s.kh, s.kt, r0, s.T, s.DH);
    fa_load<DHP, FB>(Vr, v + b * s.kb + g * s.kh, s.kt, r0, s.T, s.DH);
    auto load = [&](int it, int cur) {
        const long long hb = b * s.qb + (long long)(g * rep + it / nq) * s.qh;
        const int t = (qt0 + it % nq) * FT;
        fa_load<DHP, FT>(Qs + cur * F::TILE, q + hb, s.qt, t, s.T, s.DH);
        fa_load<DHP, FT>(Gs + cur * F::TILE, dO + hb, s.qt, t, s.T, s.DH);
    };
    if (part < n_it) load(part, 0);
    fa_commit();
    float ak[4][F::NC], av[4][F::NC];
    fa_zero(ak); fa_zero(av);
    for (int it = part, step = 0; it < n_it; it += S, step++) {
        const int cur = step & 1, h = g * rep + it / nq, q0 = (qt0 + it % nq) * FT;
        float L[4], D[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int t = q0 + kg + 8 * j;
            L[j] = t < s.T ? lse[((long long)b * s.H + h) * s.T + t] : 0.f;
            D[j] = t < s.T ? Dv[b * s.db + h * s.dh_ + (long long)t * s.dtk] : 0.f;
        }
        fa_wait();
        __syncthreads();
        if (it + S < n_it) load(it + S, cur ^ 1);
        fa_commit();
        if (q0 + FT - 1 < j0) continue;
        const float* Qt = Qs + cur * F::TILE;
        const float* Gt = Gs + cur * F::TILE;
        float sc[4][4], dp[4][4];
        fa_dot<DHP>(Kr + (warp * 16 + rg) * F::LD, Qt + kg * F::LD, s.DH, sc);
        fa_dot<DHP>(Vr + (warp * 16 + rg) * F::LD, Gt + kg * F::LD, s.DH, dp);
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int t = q0 + kg + 8 * j;
                sc[i][j] = t < s.T && t >= j0 + rg + 4 * i ? expf(sc[i][j] * s.scale - L[j]) : 0.f;
                dp[i][j] = sc[i][j] * (dp[i][j] - D[j]) * s.scale;
            }
        fa_put(P, sc, rg, kg);
        __syncwarp();
        fa_axpy<DHP>(av, P, Gt, rg, kg);
        __syncwarp();
        fa_put(P, dp, rg, kg);
        __syncwarp();
        fa_axpy<DHP>(ak, P, Qt, rg, kg);
        __syncwarp();
    }
    float* ok = dk + b * s.kb + g * s.kh;
    float* ov = dv + b * s.kb + g * s.kh;
    if (SHARE) {                         // units: dK rows, then dV rows
        fa_wait();
        __syncthreads();
        float4* x = reinterpret_cast<float4*>(smem) + threadIdx.x;
        fa_leave<F::NC>(x, ak);
        fa_leave<F::NC>(x + F::NC * FTH, av);
        cluster_sync();
        fa_of_size(S, [&](auto size) {
            constexpr int SS = decltype(size)::value;
            for (int u = part * 8 / SS; u < (part + 1) * 8 / SS; u++) {
                float a[F::NC];
                fa_gather<SS, F::NC>(x + u * (F::NC / 4) * FTH, nullptr, a);
                const int t = j0 + rg + 4 * (u & 3);
                if (t < s.T) fa_store<F::NC>((u < 4 ? ok : ov) + (long long)t * s.kt, a, 1.f, kg, s.DH);
            }
        });
        cluster_sync();                  // peers have read
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = j0 + rg + 4 * i;
        if (t >= s.T) continue;
        fa_store<F::NC>(ok + (long long)t * s.kt, ak[i], 1.f, kg, s.DH);
        fa_store<F::NC>(ov + (long long)t * s.kt, av[i], 1.f, kg, s.DH);
    }
}

// ── host ────────────────────────────────────────────────────────────────────
enum { FA_FWD, FA_DQ, FA_DKV };
template <int DHP> static constexpr int fa_smem(int which) {      // (the merge of a cluster takes less)
    return ((which == FA_FWD ? 1 : 2) * F32Att<DHP>::OWN + 4 * F32Att<DHP>::TILE + FW * F32Att<DHP>::P) * 4;
}
template <int DHP> static constexpr int fa_merge(int which) {
    return (which == FA_FWD ? 4 * (F32Att<DHP>::NC + 4) : which == FA_DQ ? 4 * F32Att<DHP>::NC : 8 * F32Att<DHP>::NC) * FTH * 4;
}
static_assert(fa_merge<32>(FA_FWD) <= fa_smem<32>(FA_FWD) && fa_merge<64>(FA_FWD) <= fa_smem<64>(FA_FWD) && fa_merge<32>(FA_DKV) <= fa_smem<32>(FA_DKV) &&
              fa_merge<64>(FA_DKV) <= fa_smem<64>(FA_DKV), "what a cluster merges takes the tiles' place");
template <int DHP> static int fa_attr() {
    int rc = 0;
    auto set = [&](auto kern, int which) { rc |= (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, fa_smem<DHP>(which)); };
    set(k_attn_fwd_f32<DHP, false>, FA_FWD); set(k_attn_fwd_f32<DHP, true>, FA_FWD);
    set(k_attn_dq_f32<DHP, false>, FA_DQ); set(k_attn_dq_f32<DHP, true>, FA_DQ);
    set(k_attn_dkv_f32<DHP, false>, FA_DKV); set(k_attn_dkv_f32<DHP, true>, FA_DKV);
    return rc;
}
int ax_attn_f32_init(void) { return fa_attr<32>() | fa_attr<64>(); }

static bool fa_served(const AttnShape& s, std::initializer_list<const void*> ptrs) {
    bool ok = s.DH > 8 && s.DH <= 64 && s.DH % 4 == 0 && s.B >= 1 && s.T >= 1 && s.KV >= 1 && s.H % s.KV == 0 && s.H <= 65535 && s.B <= 65535;
    for (long long st : {s.qb, s.qh, s.qt, s.kb, s.kh, s.kt}) ok = ok && st % 4 == 0;
    for (const void* p : ptrs) ok = ok && aligned16(p);
    return ok;
}
// CTAs that share a block's walk (powers of two, up to four, dK / dV eight), or 0: attn_simt.cu is faster, whose blocks are half as long and whose steps are shorter.
//
// The number is that of the least estimate: launch, steps of a CTA, the chip's work (steps and set-ups for each SM), which add up nearly, and a merge.  Constants are fitted to 680
// seeded shapes (T 8 to 1500, H 1 to 48; rms 10 to 12 %).  us with 1 / 2 / 4 / 8 CTAs and there (blocks, tiles of the longest walk): forward B2 H8 T256 DH32 (64, 8) 22.9 / 14.7 / 12.2
// and 14.8, B2 H16 T333 DH64 (192, 11) 65 / 41 / 40 and 63; with row dots dQ of the former 27.3 / 16.7 / 14.0 and 20.9; dK / dV of B2 H8 KV4 T256 DH32 (32, 16) 63.5 / 35.5 / 20.5 / 17.8
// and 22.8, B40 H8 KV2 T100 DH48 (160, 16) 129 / 97 / 77 / 86 and 140.  Over the 680: 0.80, 0.85 and 0.88 of the time there.
//
// There, dQ | dK / dV with row dots, here / there: sequences of one tile, which fill half a block: B240 H16 KV4 T10 DH48 104 / 73 | 124 / 86, B7 H8 KV8 T22 DH32 - | 6.5 / 6.5, B12 H24 KV12
// T14 DH16 - | 9.6 / 8.2, forward B33 H12 T17 DH32 8.9 / 7.2; few blocks with long walks, which are the latency of their steps: B1 H3 T976 DH16 32 / 24 | 51 / 41, B1 H8 KV2 T928 DH64 - | 144 / 125,
// B6 H2 KV1 T192 DH12 - | 15.1 / 11.9.
static double fa_us(int which, int DH, double walk, double work, double ctas, int S) {
    static const struct { double launch, chip, step, step_dh, step_cols, cta_col, merge, merge_col; } k[3] = {
        {1.39, 0.678, 1.33, 0.0220, 0.0141, 0.0149, 1.16, 0.0082}, {2.47, 0.767, 0.81, 0.0364, 0.0237, 0.0165, 1.45, 0.0070}, {1.83, 0.730, 1.49, 0.0342, 0.0341, 0.0450, 1.84, 0.0089}};
    const auto& c = k[which];
    const int cols = DH <= 32 ? 32 : 64;
    const double step = c.step + c.step_dh * DH + c.step_cols * cols;
    return c.launch + pow(pow(step * walk, 1.35) + pow(c.chip * step * work + c.cta_col * cols * ctas, 1.35), 1 / 1.35) + (S > 1 ? c.merge + c.merge_col * cols : 0);
}
int ax_attn_f32_ctas(int which, const AttnShape& s) {
    if (s.DH <= 8 || s.DH > 64 || s.DH % 4 || s.B < 1 || s.T < 1 || s.KV < 1 || s.H < 1 || s.H % s.KV) return 0;
    const long long nb = (s.T + FB - 1) / FB, tiles = (s.T + FT - 1) / FT, rep = s.H / s.KV, heads = (long long)(which == FA_DKV ? s.KV : s.H) * s.B;
    const long long blocks = nb * heads, chain = which == FA_DKV ? rep * tiles : tiles;
    long long work = 0;                  // tiles that all blocks of a head walk
    for (long long i = 0; i < nb; i++) work += which == FA_DKV ? rep * (tiles - i * (FB / FT)) : tiles < (i + 1) * (FB / FT) ? tiles : (i + 1) * (FB / FT);
    const bool half = s.T <= FT;         // of a block's rows
    if (which == FA_FWD && half && blocks >= 2 * AX_SMS && (s.DH > 32 || blocks < 4 * AX_SMS)) return 0;
    if (which == FA_DQ && ((half && s.DH > 32) || (blocks <= AX_SMS / 2 && chain > 8 && s.DH <= 16) || (blocks <= AX_SMS / 4 && chain > 20 && s.DH <= 32))) return 0;
    if (which == FA_DKV && ((half && (s.DH > 32 ? chain == 1 || blocks > AX_SMS : s.DH < 32 && blocks <= AX_SMS)) || (s.T > 96 && blocks < 12) ||
                            (blocks <= AX_SMS / 4 && chain > 60 && s.DH != 32) || (blocks <= 20 && chain > 8 && s.DH < 32))) return 0;
    int best = 1;
    double least = 0;
    for (int S = 1; S <= (which == FA_DKV ? 8 : 4) && S < 2 * chain; S *= 2) {
        if (S > chain && blocks * S > AX_SMS) break;     // CTAs without a tile only on SMs that have nothing else
        const double us = fa_us(which, s.DH, (double)((chain + S - 1) / S), (double)work * heads / AX_SMS, (double)blocks * S / AX_SMS, S);
        if (S == 1 || us < least) { least = us; best = S; }
    }
    return best;
}
template <typename K, typename... A>
static int fa_launch(K shared, K whole, const AttnShape& s, int heads, int smem, int S, bool early, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((s.T + FB - 1) / FB * S, heads, s.B); cfg.blockDim = dim3(FTH); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = early && ax_gemm_pdl();
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = S; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = S > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, S > 1 ? shared : whole, args..., S) == cudaSuccess ? 0 : 3;
}
template <int DHP>
static int fa_fwd(const float* q, const float* k, const float* v, float* o, float* lse, const AttnShape& s, int S, cudaStream_t st) {
    return fa_launch(k_attn_fwd_f32<DHP, true>, k_attn_fwd_f32<DHP, false>, s, s.H, fa_smem<DHP>(FA_FWD), S, true, st, q, k, v, o, lse, s);
}
template <int DHP>
static int fa_dq(const float* q, const float* k, const float* v, const float* dO, const float* lse, const float* Dv, float* dq, const AttnShape& s, int S, cudaStream_t st) {
    return fa_launch(k_attn_dq_f32<DHP, true>, k_attn_dq_f32<DHP, false>, s, s.H, fa_smem<DHP>(FA_DQ), S, true, st, q, k, v, dO, lse, Dv, dq, s);
}
template <int DHP>
static int fa_dkv(const float* q, const float* k, const float* v, const float* dO, const float* lse, const float* Dv, float* dk, float* dv, const AttnShape& s, int S, cudaStream_t st) {
    // Its CTAs come while dQ ends where they are few: 8 % of the backward with 74 and narrow heads, 3 % with wide ones; behind the larger blocks of the general dQ kernel only with 37, as
    // 74 to 111 took up to 1.4 times as long there.
    const bool early = (long long)((s.T + FB - 1) / FB) * s.KV * s.B * S <= (ax_attn_f32_ctas(FA_DQ, s) ? AX_SMS / 2 : AX_SMS / 4);
    return fa_launch(k_attn_dkv_f32<DHP, true>, k_attn_dkv_f32<DHP, false>, s, s.KV, fa_smem<DHP>(FA_DKV), S, early, st, q, k, v, dO, lse, Dv, dk, dv, s);
}
// -1: not for these kernels.  dQ and dK / dV are chosen each by itself.
int ax_attn_fwd_f32(const float* q, const float* k, const float* v, float* o, float* lse, const AttnShape& s, cudaStream_t st) {
    const int S = ax_attn_f32_ctas(FA_FWD, s);
    if (!S || !fa_served(s, {q, k, v, o})) return -1;
    ax_variant = 0x84;
    return s.DH <= 32 ? fa_fwd<32>(q, k, v, o, lse, s, S, st) : fa_fwd<64>(q, k, v, o, lse, s, S, st);
}
int ax_attn_dq_f32(const float* q, const float* k, const float* v, const float* dO, const float* lse, const float* Dv, float* dq, const AttnShape& s, cudaStream_t st) {
    const int S = ax_attn_f32_ctas(FA_DQ, s);
    if (!S || !lse || !fa_served(s, {q, k, v, dO, dq})) return -1;
    return s.DH <= 32 ? fa_dq<32>(q, k, v, dO, lse, Dv, dq, s, S, st) : fa_dq<64>(q, k, v, dO, lse, Dv, dq, s, S, st);
}
int ax_attn_dkv_f32(const float* q, const float* k, const float* v, const float* dO, const float* lse, const float* Dv, float* dk, float* dv, const AttnShape& s, cudaStream_t st) {
    const int S = ax_attn_f32_ctas(FA_DKV, s);
    if (!S || !lse || !fa_served(s, {q, k, v, dO, dk, dv})) return -1;
    return s.DH <= 32 ? fa_dkv<32>(q, k, v, dO, lse, Dv, dk, dv, s, S, st) : fa_dkv<64>(q, k, v, dO, lse, Dv, dk, dv, s, S, st);
}
