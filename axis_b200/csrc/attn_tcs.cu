// Causal grouped-query attention on tcgen05 with P and dS held to 16 bits and a sign, for head dims above 32 and up to 64 and any
// sequence length (whole tiles at head_dim 64: attn_tc.cu; other head dims: attn_tc128.cu, attn_mma.cu).  bf16, [B,T,H,DH].
//
// P and dS enter the products that take them as an operand as two bf16 numbers, hi = rn(x) and lo = rn(x - hi), in two MMAs with one
// accumulator, as in attn_mma.cu, whose comment has the errors; every sum has a fixed order, so a run repeats bit for bit.  That is
// why dQ has a kernel of its own (attn_tc.cu adds its pieces in arrival order) and computes S and dP once more.  Both numbers of an
// element fit in the 32-bit TMEM column of the score that they come from, so the second ones need no columns: they are written
// over scores that the thread has in registers, and the next scores for those columns wait for the product that reads them.
// Tiles that overhang the sequence or a narrower head are zero-filled by TMA and clipped by the stores.
//
//   forward   CTA: 128 queries of a head, two CTAs per SM (256 TMEM columns: S 128, P hi 64, O 64; P lo over S)
//   dQ        CTA: 128 queries of a head, two CTAs per SM; 64 keys a step; Q and dO in TMEM as A operands (256 columns: S and dP 64
//             each, dQ 64, Q 32, dO 32; dS over the scores; S and dP change places at each step, so that S of the next step, which
//             the exponentials need first, runs beside the dQ product)
//   dK / dV   CTA: 128 keys of a kv head, 64 queries a step; K and V in TMEM, S^T and dP^T doubled (448 columns), P^T and dS^T in
//             place; issuing warps for the scores, dV and dK, sixteen softmax warps in two groups that take the steps in turn
//
// Bound by the softmax warps: the schedulers issue in 37 % (forward), 38 % (dQ) and 46 % (dK / dV) of the cycles, the XU pipe (exponentials) is busy
// 37, 30 and 25 % (B3 H24 KV8 T1000 DH64: 34, 42 and 66 us); what is left of a step is the round trip MMA -> TMEM load -> MMA, which two CTAs or two groups cover in part.
// Forward / backward with the row dots in us, mma.sync -> here (one cold launch each): B3 H24 KV8 T1000 DH64 70 / 203 -> 36 / 106,
// B4 H24 KV8 T500 DH64 33 / 102 -> 22 / 60, B1 H12 KV4 T2500 DH64 88 / 225 -> 46 / 137, B8 H24 KV8 T320 DH64 29 / 85 -> 25 / 52.
#include "common.cuh"
#include "kernels.h"
#include "tc_common.cuh"
#include "attn_common.cuh"

#define XT 128                 // queries / keys per tile
#define XD 64                  // columns of a tile (narrower heads are zero-filled)
#define XQ 64                  // keys (dQ) or queries (dK / dV) per step
#define STAT_XFWD 0x900
#define STAT_XDQ 0xa00
#define STAT_XDKV 0xb00

// the same for a thread's columns c0 .. c0 + 15 and c0 + 32 .. c0 + 47 of an accumulator in TMEM
__device__ __forceinline__ void store_grad_row(uint32_t taddr, int c0, float f, const float* cr, const float* sr, bf16* row, int dh, bool live) {
    uint32_t v1[16], v2[16];
    tmem_ld16(taddr + c0, v1);
    tmem_ld16(taddr + 32 + c0, v2);
    tmem_ld_wait();
    if (!live) return;
#pragma unroll
    for (int q = 0; q < 16; q += 8) store_grad8(reinterpret_cast<float*>(v1 + q), reinterpret_cast<float*>(v2 + q), c0 + q, f, cr, sr, row, dh);
}
// half (32 columns, 64 bytes) of a 128-byte swizzled shared-memory row into 16 TMEM columns
__device__ __forceinline__ void row_to_tmem(const uint8_t* tile, int r, int hc, uint32_t taddr) {
    uint32_t w[16];
#pragma unroll
    for (int c4 = 0; c4 < 4; c4++) {
        const uint4 x = *reinterpret_cast<const uint4*>(tile + r * 128 + (((hc * 4 + c4) ^ (r & 7)) << 4));
        w[c4 * 4] = x.x; w[c4 * 4 + 1] = x.y; w[c4 * 4 + 2] = x.z; w[c4 * 4 + 3] = x.w;
    }
    tmem_st16(taddr + hc * 16, w);
}

// ════════════════════════════════ forward ═══════════════════════════════════
#define XF_THREADS 160         // 4 softmax warps + 1 control warp
struct XFwdSmem {
    static constexpr int Q = 0, K0 = 16384, V0 = K0 + 2 * 16384, BARS = V0 + 2 * 16384, TOTAL = BARS + 128 + 1024;
};
__global__ void __launch_bounds__(XF_THREADS, 2)
k_attn_fwd_tcs(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
               bf16* __restrict__ o, float* __restrict__ lse, int T, int H, int KV, int dh, float scale, int* status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sb = smem_u32(smem);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + XFwdSmem::BARS);
    // q_full, k_full[2], v_full[2], s_full, p_full, o_done
    const uint32_t b_q = smem_u32(bars), b_kf = b_q + 8, b_vf = b_kf + 16, b_s = b_vf + 16, b_p = b_s + 8, b_o = b_p + 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // 1-D grid by decreasing work: the last query tile of every (head, batch) first
    const int nqt = (T + XT - 1) / XT, nhb = gridDim.x / nqt;
    const int qt = nqt - 1 - (int)(blockIdx.x / nhb), hb = blockIdx.x % nhb;
    const int h = hb % H, b = hb / H, g = h / (H / KV);
    const int nkt = qt + 1;

    if (threadIdx.x == 0) {
        mbar_init(b_q, 1);
        for (int s = 0; s < 2; s++) { mbar_init(b_kf + 8 * s, 1); mbar_init(b_vf + 8 * s, 1); }
        mbar_init(b_s, 1); mbar_init(b_p, 128); mbar_init(b_o, 1);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 4) { tmem_alloc(smem_u32(tmem_slot), 256); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t t_S = tmem, t_P = tmem + 128, t_O = tmem + 192;
    pdl_enter();

    if (warp == 4) {
        bool ok = true;
        constexpr uint32_t id_s = tc_idesc_bf16(128, 128, 0, 0), id_pv = tc_idesc_bf16(128, 64, 0, 1);
        const uint32_t loQ = desc_lo(sb + XFwdSmem::Q, 16), loK = desc_lo(sb + XFwdSmem::K0, 16), loV = desc_lo(sb + XFwdSmem::V0, 16384);
        auto load = [&](const CUtensorMap* m, uint32_t bar, int at, int j) {
            if (lane == 0) {
                mbar_expect_tx(bar + 8 * (j & 1), 16384);
                tma_load_4d(sb + at + (j & 1) * 16384, m, bar + 8 * (j & 1), 0, g, j * XT, b);
            }
        };
        auto issue_s = [&](int j) {
#pragma unroll
            for (int kk = 0; kk < XD / 16; kk++)
                mma_ss_e(t_S, desc_of(loQ + kk * 2), desc_of(loK + (j & 1) * 1024 + kk * 2), id_s, kk != 0);
            commit_e(b_s);
        };
        if (lane == 0) {
            mbar_expect_tx(b_q, 16384);
            tma_load_4d(sb + XFwdSmem::Q, &tmQ, b_q, 0, h, qt * XT, b);
        }
        for (int j = 0; j < 2 && j < nkt; j++) { load(&tmK, b_kf, XFwdSmem::K0, j); load(&tmV, b_vf, XFwdSmem::V0, j); }
        __syncwarp();
        if (!mbar_wait_park(b_q, 0) || !mbar_wait_park(b_kf, 0)) ok = false;
        if (ok) { tc_fence_after(); issue_s(0); }
        for (int j = 0; j < nkt && ok; j++) {
            const int s = j & 1;
            // O += P(j) V(j): the second numbers (columns of S), then the first
            if (!mbar_wait_park(b_vf + 8 * s, (j >> 1) & 1) || !mbar_wait_park(b_p, j & 1) || *abort_flag) { ok = false; break; }
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < XT / 16; kk++)
                mma_ts_e(t_O, t_S + kk * 8, desc_of(loV + s * 1024 + kk * 128), id_pv, (j | kk) != 0);
#pragma unroll
            for (int kk = 0; kk < XT / 16; kk++)
                mma_ts_e(t_O, t_P + kk * 8, desc_of(loV + s * 1024 + kk * 128), id_pv, 1);
            commit_e(b_o);
            if (j + 2 < nkt) { load(&tmK, b_kf, XFwdSmem::K0, j + 2); __syncwarp(); }     // S(j) has run: its result was read
            if (j + 1 < nkt) {
                if (!mbar_wait_park(b_kf + 8 * (s ^ 1), ((j + 1) >> 1) & 1) || !mbar_wait_park(b_o, j & 1)) { ok = false; break; }
                tc_fence_after();
                issue_s(j + 1);
                if (j + 2 < nkt) { load(&tmV, b_vf, XFwdSmem::V0, j + 2); __syncwarp(); }
            }
        }
        __syncwarp();
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(status, STAT_XFWD | 1); }
    } else {
        const int r = threadIdx.x;                         // query row within the tile == TMEM lane
        const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
        const float c = scale * LOG2E;
        const float2 c2 = make_float2(c, c);
        float m_used = -INFINITY, l = 0.f;
        bool ok = true;
        for (int j = 0; j < nkt && ok; j++) {
            // S(j) was issued behind the commit of P(j-1) V(j-1): the P and O columns are free as well
            if (!mbar_wait_park(b_s, j & 1) || *abort_flag) { ok = false; break; }
            tc_fence_after();
            uint32_t sv[128];
#pragma unroll
            for (int ch = 0; ch < 4; ch++) tmem_ld32(t_S + lane_base + ch * 32, sv + ch * 32);
            tmem_ld_wait();
            if (j == qt) {
#pragma unroll
                for (int q = 0; q < 128; q++)
                    if (q > r) sv[q] = 0xff800000u;              // -inf: exp2 gives 0
            }
            float mx;
            {
                float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
                for (int q = 0; q < 128; q += 8) {
                    m0 = fmax3(m0, __uint_as_float(sv[q]), __uint_as_float(sv[q + 1]));
                    m1 = fmax3(m1, __uint_as_float(sv[q + 2]), __uint_as_float(sv[q + 3]));
                    m2 = fmax3(m2, __uint_as_float(sv[q + 4]), __uint_as_float(sv[q + 5]));
                    m3 = fmax3(m3, __uint_as_float(sv[q + 6]), __uint_as_float(sv[q + 7]));
                }
                mx = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3)) * c;
            }
            if (j == 0) {
                m_used = mx;
            } else if (__any_sync(0xffffffffu, mx > m_used + 8.f)) {
                const float m_new = fmaxf(m_used, mx);
                const float f = fast_exp2(m_used - m_new);
                m_used = m_new;
                l *= f;
#pragma unroll 1
                for (int ch = 0; ch < 4; ch++) {
                    uint32_t v[16];
                    tmem_ld16(t_O + lane_base + ch * 16, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int q = 0; q < 16; q++) v[q] = __float_as_uint(__uint_as_float(v[q]) * f);
                    tmem_st16(t_O + lane_base + ch * 16, v);
                }
            }
            const float2 nm2 = make_float2(-m_used, -m_used);
            float2 l2 = make_float2(0.f, 0.f);
#pragma unroll
            for (int ch = 0; ch < 4; ch++) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int q = 0; q < 32; q += 2) {
                    const float2 x = __ffma2_rn(make_float2(__uint_as_float(sv[ch * 32 + q]), __uint_as_float(sv[ch * 32 + q + 1])), c2, nm2);
                    const float2 p = make_float2(fast_exp2(x.x), fast_exp2(x.y));
                    l2 = __fadd2_rn(l2, p);
                    split_bf16(p.x, p.y, hi[q >> 1], lo[q >> 1]);
                }
                tmem_st16(t_P + lane_base + ch * 16, hi);
                tmem_st16(t_S + lane_base + ch * 16, lo);
            }
            l += l2.x + l2.y;
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(b_p);
        }
        if (ok && mbar_wait_park(b_o, (nkt - 1) & 1)) {
            tc_fence_after();
            const int t = qt * XT + r;
            const float il = 1.f / l;
            bf16* orow = o + (((long long)b * T + t) * H + h) * dh;
#pragma unroll 1
            for (int ch = 0; ch < 2; ch++) {
                uint32_t v[32];
                tmem_ld32(t_O + lane_base + ch * 32, v);
                tmem_ld_wait();
                if (t < T) {
#pragma unroll
                    for (int q = 0; q < 32; q += 8) {
                        uint4 pk;
                        pk.x = pack_bf16(__uint_as_float(v[q]) * il, __uint_as_float(v[q + 1]) * il);
                        pk.y = pack_bf16(__uint_as_float(v[q + 2]) * il, __uint_as_float(v[q + 3]) * il);
                        pk.z = pack_bf16(__uint_as_float(v[q + 4]) * il, __uint_as_float(v[q + 5]) * il);
                        pk.w = pack_bf16(__uint_as_float(v[q + 6]) * il, __uint_as_float(v[q + 7]) * il);
                        if (ch * 32 + q < dh) *reinterpret_cast<uint4*>(orow + ch * 32 + q) = pk;
                    }
                }
            }
            if (t < T) lse[((long long)b * H + h) * T + t] = (m_used + log2f(l)) * LN2;
        } else if (lane == 0) {
            *abort_flag = 1;
            atomicExch(status, STAT_XFWD | 2);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 4) { __syncwarp(); tc_fence_after(); tmem_dealloc(tmem, 256); }
}

// ════════════════════════════════ dQ ════════════════════════════════════════
#define XG_THREADS 288         // 8 softmax warps (lane quarter, column half) + 1 control warp
#define XG_SLOTS 3             // K / V ring
struct XdQSmem {
    static constexpr int Q = 0, DO = 16384, K0 = 32768, V0 = K0 + XG_SLOTS * 8192, BARS = V0 + XG_SLOTS * 8192, TOTAL = BARS + 128 + 1024;
};
__global__ void __launch_bounds__(XG_THREADS, 2)
k_attn_dq_tcs(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO, const __grid_constant__ CUtensorMap tmK,
              const __grid_constant__ CUtensorMap tmV, const float* __restrict__ lse, const float* __restrict__ Dv, bf16* __restrict__ dq,
              const AttnShape s, const float* __restrict__ rope_cos, const float* __restrict__ rope_sin, int* status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sb = smem_u32(smem);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + XdQSmem::BARS);
    // q_full, q_in_tmem, kv_full[3], s_full, dp_full, ds_full, dq_done
    const uint32_t b_q = smem_u32(bars), b_qt = b_q + 8, b_kv = b_qt + 8, b_s = b_kv + 8 * XG_SLOTS, b_dp = b_s + 8, b_ds = b_dp + 8, b_o = b_ds + 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 12);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int T = s.T, H = s.H, nqt = (T + XT - 1) / XT, nhb = gridDim.x / nqt;
    const int qt = nqt - 1 - (int)(blockIdx.x / nhb), hb = blockIdx.x % nhb;
    const int h = hb % H, b = hb / H, g = h / (H / s.KV);
    const int n = min(2 * (qt + 1), (T + XQ - 1) / XQ);       // steps

    if (threadIdx.x == 0) {
        mbar_init(b_q, 1); mbar_init(b_qt, 256);
        for (int i = 0; i < XG_SLOTS; i++) mbar_init(b_kv + 8 * i, 1);
        mbar_init(b_s, 1); mbar_init(b_dp, 1); mbar_init(b_ds, 256); mbar_init(b_o, 1);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 8) { tmem_alloc(smem_u32(tmem_slot), 256); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t t_X = tmem, t_dQ = tmem + 128, t_Q = tmem + 192, t_G = tmem + 224;      // X: two regions, S and dP in turn
    pdl_enter();

    if (warp == 8) {
        bool ok = true;
        constexpr uint32_t id_s = tc_idesc_bf16(128, 64, 0, 0), id_dq = tc_idesc_bf16(128, 64, 0, 1);
        const uint32_t loK = desc_lo(sb + XdQSmem::K0, 16), loV = desc_lo(sb + XdQSmem::V0, 16), loKn = desc_lo(sb + XdQSmem::K0, 16384);
        auto load = [&](int j) {
            if (lane == 0) {
                const int sl = j % XG_SLOTS;
                mbar_expect_tx(b_kv + 8 * sl, 16384);
                tma_load_4d(sb + XdQSmem::K0 + sl * 8192, &tmK, b_kv + 8 * sl, 0, g, j * XQ, b);
                tma_load_4d(sb + XdQSmem::V0 + sl * 8192, &tmV, b_kv + 8 * sl, 0, g, j * XQ, b);
            }
        };
        auto issue = [&](uint32_t d, uint32_t a, uint32_t lo, int j, uint32_t bar) {
#pragma unroll
            for (int kk = 0; kk < XD / 16; kk++) mma_ts_e(d, a + kk * 8, desc_of(lo + (j % XG_SLOTS) * 512 + kk * 2), id_s, kk != 0);
            commit_e(bar);
        };
        if (lane == 0) {
            mbar_expect_tx(b_q, 32768);
            tma_load_4d(sb + XdQSmem::Q, &tmQ, b_q, 0, h, qt * XT, b);
            tma_load_4d(sb + XdQSmem::DO, &tmdO, b_q, 0, h, qt * XT, b);
        }
        for (int j = 0; j < XG_SLOTS && j < n; j++) load(j);
        __syncwarp();
        if (!mbar_wait_park(b_qt, 0) || !mbar_wait_park(b_kv, 0)) ok = false;
        tc_fence_after();
        if (ok) { issue(t_X, t_Q, loK, 0, b_s); issue(t_X + 64, t_G, loV, 0, b_dp); }
        for (int j = 0; j < n && ok; j++) {
            const uint32_t x = t_X + (j & 1) * 64, y = t_X + (~j & 1) * 64;      // S(j), now dS(j); dP(j), read
            if (!mbar_wait_park(b_ds, j & 1) || *abort_flag) { ok = false; break; }
            if (j + 1 < n && !mbar_wait_park(b_kv + 8 * ((j + 1) % XG_SLOTS), ((j + 1) / XG_SLOTS) & 1)) { ok = false; break; }
            tc_fence_after();
            if (j + 1 < n) issue(y, t_Q, loK, j + 1, b_s);
            // dQ += dS(j) K(j): sixteen keys are eight packed columns; of a thread's 32 columns the first 16 hold the first numbers
#pragma unroll
            for (int i = 1; i >= 0; i--)
#pragma unroll
                for (int kk = 0; kk < XQ / 16; kk++)
                    mma_ts_e(t_dQ, x + (kk >> 1) * 32 + i * 16 + (kk & 1) * 8, desc_of(loKn + (j % XG_SLOTS) * 512 + kk * 128), id_dq, (j | (i ^ 1) | kk) != 0);
            commit_e(b_o);
            if (j + 1 < n) {
                if (!mbar_wait_park(b_o, j & 1)) { ok = false; break; }
                tc_fence_after();
                issue(x, t_G, loV, j + 1, b_dp);
                if (j + XG_SLOTS < n) { load(j + XG_SLOTS); __syncwarp(); }
            }
        }
        __syncwarp();
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(status, STAT_XDQ | 1); }
    } else {
        const int r = threadIdx.x & 127, hc = warp >> 2;            // query row == TMEM lane; column half
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        const int t = qt * XT + r;
        const float c = s.scale * LOG2E;
        const float L = t < T ? -lse[((long long)b * H + h) * T + t] * LOG2E : -INFINITY;      // a row past T: P = 0
        const float D = t < T ? -Dv[b * s.db + h * s.dh_ + t * s.dtk] : 0.f;
        const float2 c2 = make_float2(c, c), L2 = make_float2(L, L), D2 = make_float2(D, D);
        bool ok = mbar_wait_park(b_q, 0);
        if (ok) {
            row_to_tmem(smem + XdQSmem::Q, r, hc, t_Q + lane_base);
            row_to_tmem(smem + XdQSmem::DO, r, hc, t_G + lane_base);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(b_qt);
        }
        for (int j = 0; j < n && ok; j++) {
            const uint32_t x = t_X + (j & 1) * 64 + hc * 32 + lane_base, y = t_X + (~j & 1) * 64 + hc * 32 + lane_base;
            if (!mbar_wait_park(b_s, j & 1) || *abort_flag) { ok = false; break; }
            tc_fence_after();
            uint32_t sv[32], dp[32];
            tmem_ld32(x, sv);
            tmem_ld_wait();
            if (j >= 2 * qt) {                                      // the diagonal: keys behind the query
                const int last = t - j * XQ - hc * 32;
#pragma unroll
                for (int q = 0; q < 32; q++)
                    if (q > last) sv[q] = 0xff800000u;
            }
#pragma unroll
            for (int q = 0; q < 32; q += 2) {
                const float2 e = __ffma2_rn(make_float2(__uint_as_float(sv[q]), __uint_as_float(sv[q + 1])), c2, L2);
                sv[q] = __float_as_uint(fast_exp2(e.x)); sv[q + 1] = __float_as_uint(fast_exp2(e.y));
            }
            if (!mbar_wait_park(b_dp, j & 1)) { ok = false; break; }
            tc_fence_after();
            tmem_ld32(y, dp);
            tmem_ld_wait();
            uint32_t hi[16], lo[16];
#pragma unroll
            for (int q = 0; q < 32; q += 2) {
                const float2 e = __fadd2_rn(make_float2(__uint_as_float(dp[q]), __uint_as_float(dp[q + 1])), D2);
                const float2 d = __fmul2_rn(make_float2(__uint_as_float(sv[q]), __uint_as_float(sv[q + 1])), e);
                split_bf16(d.x, d.y, hi[q >> 1], lo[q >> 1]);
            }
            tmem_st16(x, hi);
            tmem_st16(x + 16, lo);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(b_ds);
        }
        if (ok && mbar_wait_park(b_o, (n - 1) & 1)) {
            tc_fence_after();
            store_grad_row(t_dQ + lane_base, hc * 16, s.scale, rope_cos ? rope_cos + (long long)t * 32 : nullptr, rope_sin + (long long)t * 32,
                           dq + (((long long)b * T + t) * H + h) * s.DH, s.DH, t < T);
        } else if (lane == 0) {
            *abort_flag = 1;
            atomicExch(status, STAT_XDQ | 2);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 8) { __syncwarp(); tc_fence_after(); tmem_dealloc(tmem, 256); }
}

// ════════════════════════════════ dK, dV ════════════════════════════════════
#define XK_SM_WARPS 16
#define XK_THREADS ((XK_SM_WARPS + 4) * 32)
#define XK_SLOTS 5
struct XdKVSmem {
    static constexpr int K = 0, V = 16384, Q0 = 32768, DO0 = Q0 + XK_SLOTS * 8192, STAT = DO0 + XK_SLOTS * 8192, MINE = STAT + XK_SLOTS * 512,
                         BARS = MINE + XK_SM_WARPS * 256, TOTAL = BARS + 256 + 1024;
};
// Warp 16 + i: 0 S^T = K Q^T and dP^T = V dO^T, 1 dV += P^T dO, 2 dK += dS^T Q, 3 loads (Q and dO by TMA, lse and D by lanes, since rows
// of any T have no alignment).  Softmax group e = warp / 8 takes the steps of parity e; in it a warp has a lane quarter (32 keys) and
// half of the 64 query columns.
// A cluster of S CTAs takes the steps of a key tile in turn where one chain would be the kernel (see the launch); their sums meet
// through distributed shared memory in rank order, each CTA finishing 128 / S of the rows.
#define XK_PITCH 68            // floats of a row of sums: rows of a warp fall in different banks
static_assert(2 * XT * XK_PITCH * 4 <= 2 * XK_SLOTS * 8192, "the sums take the ring's place");
__global__ void __launch_bounds__(XK_THREADS, 1)
k_attn_dkv_tcs(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO, const __grid_constant__ CUtensorMap tmK,
               const __grid_constant__ CUtensorMap tmV, const float* __restrict__ lse, const float* __restrict__ Dv, bf16* __restrict__ dk,
               bf16* __restrict__ dv, const AttnShape s, int S, const float* __restrict__ rope_cos, const float* __restrict__ rope_sin, int* status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sb = smem_u32(smem);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + XdKVSmem::BARS);
    // kv_full, kv_in_tmem, q_full[5], q_empty[5], sdp_full[2], pds_full[2]
    const uint32_t b_kv = smem_u32(bars), b_kvt = b_kv + 8, b_qf = b_kvt + 8, b_qe = b_qf + 8 * XK_SLOTS, b_s = b_qe + 8 * XK_SLOTS, b_pds = b_s + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 24);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* stat = reinterpret_cast<float*>(smem + XdKVSmem::STAT);        // [slot][-lse log2(e) 64 | -D 64]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // 1-D grid by decreasing work: key tile 0, which every query attends to, of all (kv head, batch) first
    const int T = s.T, H = s.H, KV = s.KV, rep = H / KV, ngb = KV * s.B;
    const int part = blockIdx.x % S, tile = blockIdx.x / S, j = tile / ngb, gb = tile % ngb, g = gb % KV, b = gb / KV;
    const int nq = (T + XQ - 1) / XQ, per = nq - 2 * j;                   // 64-query steps per head
    const int n = (rep * per - part + S - 1) / S;                         // this CTA's: part, part + S, ... of all heads'

    if (threadIdx.x == 0) {
        mbar_init(b_kv, 1); mbar_init(b_kvt, XK_SM_WARPS * 32);
        for (int i = 0; i < XK_SLOTS; i++) { mbar_init(b_qf + 8 * i, 33); mbar_init(b_qe + 8 * i, 2); }
        for (int i = 0; i < 2; i++) { mbar_init(b_s + 8 * i, 1); mbar_init(b_pds + 8 * i, 256); }
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == XK_SM_WARPS) { tmem_alloc(smem_u32(tmem_slot), 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t t_S = tmem, t_dP = tmem + 128, t_dV = tmem + 256, t_dK = tmem + 320, t_K = tmem + 384, t_V = tmem + 416;
    pdl_enter();

    if (warp == XK_SM_WARPS + 3) {
        bool ok = true;
        if (lane == 0) {
            mbar_expect_tx(b_kv, 32768);
            tma_load_4d(sb + XdKVSmem::K, &tmK, b_kv, 0, g, j * XT, b);
            tma_load_4d(sb + XdKVSmem::V, &tmV, b_kv, 0, g, j * XT, b);
        }
        __syncwarp();
        int sl = 0, ph = 0, hh = 0, qi = 2 * j + part;
        for (int u = 0; u < n && ok; u++) {
            while (qi >= nq) { qi -= per; hh++; }
            const int h = g * rep + hh, t0 = qi * XQ;
            float st[2][2];                                   // of rows t0 + lane, t0 + lane + 32; a row past T: P = 0
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int t = t0 + i * 32 + lane;
                st[0][i] = t < T ? -lse[((long long)b * H + h) * T + t] * LOG2E : -INFINITY;
                st[1][i] = t < T ? -Dv[b * s.db + h * s.dh_ + t * s.dtk] : 0.f;
            }
            if (u >= XK_SLOTS && (!mbar_wait_park(b_qe + 8 * sl, ph ^ 1) || *abort_flag)) { ok = false; break; }
            if (lane == 0) {
                mbar_expect_tx(b_qf + 8 * sl, 16384);
                tma_load_4d(sb + XdKVSmem::Q0 + sl * 8192, &tmQ, b_qf + 8 * sl, 0, h, t0, b);
                tma_load_4d(sb + XdKVSmem::DO0 + sl * 8192, &tmdO, b_qf + 8 * sl, 0, h, t0, b);
            }
#pragma unroll
            for (int i = 0; i < 4; i++) stat[sl * 128 + i * 32 + lane] = st[i >> 1][i & 1];
            mbar_arrive(b_qf + 8 * sl);
            if (++sl == XK_SLOTS) { sl = 0; ph ^= 1; }
            qi += S;
        }
        __syncwarp();
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(status, STAT_XDKV | 3); }
    } else if (warp > XK_SM_WARPS) {
        const bool is_v = warp == XK_SM_WARPS + 1;
        bool ok = true;
        constexpr uint32_t id_acc = tc_idesc_bf16(128, 64, 0, 1);      // A in TMEM, B N-major
        const uint32_t loB = is_v ? desc_lo(sb + XdKVSmem::DO0, 16384) : desc_lo(sb + XdKVSmem::Q0, 16384);
        const uint32_t tA = is_v ? t_S : t_dP, tD = is_v ? t_dV : t_dK;
        int sl = 0;
        for (int u = 0; u < n && ok; u++) {
            const int e = u & 1;
            if (!mbar_wait_park(b_pds + 8 * e, (u >> 1) & 1) || *abort_flag) { ok = false; break; }
            tc_fence_after();
            // sixteen queries: eight packed columns of first numbers, then eight of second ones
#pragma unroll
            for (int i = 1; i >= 0; i--)
#pragma unroll
                for (int kk = 0; kk < XQ / 16; kk++)
                    mma_ts_e(tD, tA + e * 64 + kk * 16 + i * 8, desc_of(loB + (uint32_t)sl * 512 + kk * 128), id_acc, (u | (i ^ 1) | kk) != 0);
            commit_e(b_qe + 8 * sl);                   // two arrivals (dV and dK): the ring slot and both buffers are free
            if (++sl == XK_SLOTS) sl = 0;
        }
        __syncwarp();
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(status, STAT_XDKV | 4); }
    } else if (warp == XK_SM_WARPS) {
        bool ok = mbar_wait_park(b_kvt, 0);                   // K and V are in TMEM
        constexpr uint32_t id_s = tc_idesc_bf16(128, 64, 0, 0);
        const uint32_t loQ = desc_lo(sb + XdKVSmem::Q0, 16), loG = desc_lo(sb + XdKVSmem::DO0, 16);
        tc_fence_after();
        int sl = 0, ph = 0, sl_p = 0, ph_p = 0;         // ring slot and parity of step u; of step u - 2
        for (int u = 0; u < n && ok; u++) {
            if (!mbar_wait_park(b_qf + 8 * sl, ph) || *abort_flag) { ok = false; break; }
            // dV / dK(u-2) have read P^T / dS^T out of the two buffers that S^T / dP^T(u) overwrite
            if (u >= 2) {
                if (!mbar_wait_park(b_qe + 8 * sl_p, ph_p)) { ok = false; break; }
                if (++sl_p == XK_SLOTS) { sl_p = 0; ph_p ^= 1; }
            }
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < XD / 16; kk++)
                mma_ts_e(t_S + (u & 1) * 64, t_K + kk * 8, desc_of(loQ + (uint32_t)sl * 512 + kk * 2), id_s, kk != 0);
#pragma unroll
            for (int kk = 0; kk < XD / 16; kk++)
                mma_ts_e(t_dP + (u & 1) * 64, t_V + kk * 8, desc_of(loG + (uint32_t)sl * 512 + kk * 2), id_s, kk != 0);
            commit_e(b_s + 8 * (u & 1));
            if (++sl == XK_SLOTS) { sl = 0; ph ^= 1; }
        }
        __syncwarp();
        if (!ok && lane == 0) { *abort_flag = 1; atomicExch(status, STAT_XDKV | 1); }
    } else {
        const int r = threadIdx.x & 127, e = warp >> 3, hc = (warp >> 2) & 1;     // key row == TMEM lane; group; column half
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        const float c = s.scale * LOG2E;
        const float2 c2 = make_float2(c, c);
        float* mine = reinterpret_cast<float*>(smem + XdKVSmem::MINE) + warp * 64;  // the warp's columns of the step's statistics
        bool ok = mbar_wait_park(b_kv, 0);
        if (ok) {
            row_to_tmem(smem + (e ? XdKVSmem::V : XdKVSmem::K), r, hc, (e ? t_V : t_K) + lane_base);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(b_kvt);
        }
        int sl = e, ph = 0, qi = 2 * j + part + e * S;
        for (int u = e; u < n && ok; u += 2) {
            while (qi >= nq) qi -= per;
            if (!mbar_wait_park(b_s + 8 * e, (u >> 1) & 1) || *abort_flag) { ok = false; break; }
            if (!mbar_wait_park(b_qf + 8 * sl, ph)) { ok = false; break; }         // complete since S^T was issued: makes the statistics visible
            tc_fence_after();
            mine[lane] = stat[sl * 128 + hc * 32 + lane];
            mine[32 + lane] = stat[sl * 128 + 64 + hc * 32 + lane];
            __syncwarp();
            const uint32_t tS = t_S + e * 64 + hc * 32 + lane_base, tdP = t_dP + e * 64 + hc * 32 + lane_base;
            const int first = j * XT + r - qi * XQ - hc * 32;                     // column of the key's own query
#pragma unroll
            for (int rd = 0; rd < 2; rd++) {
                uint32_t sv[16], dp[16], w[16], wd[16];
                tmem_ld16(tS + rd * 16, sv);
                tmem_ld16(tdP + rd * 16, dp);
                tmem_ld_wait();
                if (qi < 2 * j + 2) {                            // the diagonal: queries before the key
#pragma unroll
                    for (int q = 0; q < 16; q++)
                        if (rd * 16 + q < first) sv[q] = 0xff800000u;
                }
#pragma unroll
                for (int q = 0; q < 16; q += 4) {
                    const float4 l4 = *reinterpret_cast<const float4*>(mine + rd * 16 + q);       // broadcast loads
                    const float4 d4 = *reinterpret_cast<const float4*>(mine + 32 + rd * 16 + q);
                    const float2 x01 = __ffma2_rn(make_float2(__uint_as_float(sv[q]), __uint_as_float(sv[q + 1])), c2, make_float2(l4.x, l4.y));
                    const float2 x23 = __ffma2_rn(make_float2(__uint_as_float(sv[q + 2]), __uint_as_float(sv[q + 3])), c2, make_float2(l4.z, l4.w));
                    const float2 p01 = make_float2(fast_exp2(x01.x), fast_exp2(x01.y)), p23 = make_float2(fast_exp2(x23.x), fast_exp2(x23.y));
                    const float2 g01 = __fadd2_rn(make_float2(__uint_as_float(dp[q]), __uint_as_float(dp[q + 1])), make_float2(d4.x, d4.y));
                    const float2 g23 = __fadd2_rn(make_float2(__uint_as_float(dp[q + 2]), __uint_as_float(dp[q + 3])), make_float2(d4.z, d4.w));
                    const float2 s01 = __fmul2_rn(p01, g01), s23 = __fmul2_rn(p23, g23);
                    split_bf16(p01.x, p01.y, w[q >> 1], w[8 + (q >> 1)]);
                    split_bf16(p23.x, p23.y, w[(q >> 1) + 1], w[9 + (q >> 1)]);
                    split_bf16(s01.x, s01.y, wd[q >> 1], wd[8 + (q >> 1)]);
                    split_bf16(s23.x, s23.y, wd[(q >> 1) + 1], wd[9 + (q >> 1)]);
                }
                tmem_st16(tS + rd * 16, w);                     // the columns that this round has read
                tmem_st16(tdP + rd * 16, wd);
            }
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(b_pds + 8 * e);
            sl += 2;
            if (sl >= XK_SLOTS) { sl -= XK_SLOTS; ph ^= 1; }
            qi += 2 * S;
            __syncwarp();                                    // the warp's statistics are rewritten
        }
        // dV (group 0) and dK (group 1)
        if (ok && (n == 0 || mbar_wait_park(b_qe + 8 * ((n - 1) % XK_SLOTS), ((n - 1) / XK_SLOTS) & 1))) {
            tc_fence_after();
            const int t = j * XT + r;
            if (S > 1) {                                     // [dV, dK][key][64], in the ring's place: its last reader has run
                float* row = reinterpret_cast<float*>(smem + XdKVSmem::Q0) + (e * XT + r) * XK_PITCH + hc * 32;
                uint32_t v[32];
                if (n) {
                    tmem_ld32((e ? t_dK : t_dV) + lane_base + hc * 32, v);
                    tmem_ld_wait();
                }
#pragma unroll
                for (int q = 0; q < 32; q += 4)
                    *reinterpret_cast<uint4*>(row + q) = n ? make_uint4(v[q], v[q + 1], v[q + 2], v[q + 3]) : make_uint4(0, 0, 0, 0);
            } else {
                store_grad_row((e ? t_dK : t_dV) + lane_base, hc * 16, e ? s.scale : 1.f, e && rope_cos ? rope_cos + (long long)t * 32 : nullptr,
                               rope_sin + (long long)t * 32, (e ? dk : dv) + (((long long)b * T + t) * KV + g) * s.DH, s.DH, t < T);
            }
        } else if (lane == 0) {
            *abort_flag = 1;
            atomicExch(status, STAT_XDKV | 2);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == XK_SM_WARPS) { __syncwarp(); tc_fence_after(); tmem_dealloc(tmem, 512); }
    if (S > 1) {
        cluster_sync();
        const int rows = XT / S;
        for (int i = threadIdx.x; i < 2 * rows * 4; i += XK_THREADS) {       // eight columns and their partners
            const int m = i / (rows * 4), r = part * rows + (i >> 2) % rows, c0 = (i & 3) * 8, t = j * XT + r;
            if (t >= T) continue;
            const uint32_t at = sb + XdKVSmem::Q0 + ((m * XT + r) * XK_PITCH + c0) * 4;
            float a[16];
            cluster_sum16<32>(at, S, a);
            store_grad8(a, a + 8, c0, m ? s.scale : 1.f, m && rope_cos ? rope_cos + (long long)t * 32 : nullptr, rope_sin + (long long)t * 32,
                        (m ? dk : dv) + (((long long)b * T + t) * KV + g) * s.DH, s.DH);
        }
        cluster_sync();     // peers have read
    }
}

// ── host ────────────────────────────────────────────────────────────────────
int ax_attn_tcs_init(void) {
    int rc = (int)cudaFuncSetAttribute(k_attn_fwd_tcs, cudaFuncAttributeMaxDynamicSharedMemorySize, XFwdSmem::TOTAL);
    rc |= (int)cudaFuncSetAttribute(k_attn_dq_tcs, cudaFuncAttributeMaxDynamicSharedMemorySize, XdQSmem::TOTAL);
    return rc | (int)cudaFuncSetAttribute(k_attn_dkv_tcs, cudaFuncAttributeMaxDynamicSharedMemorySize, XdKVSmem::TOTAL);
}
static bool served(const AttnShape& s) {
    // a positive scale: a masked score of -inf times any other is NaN or +inf
    return s.scale > 0.f && s.DH > 32 && s.DH <= XD && s.DH % 8 == 0 && s.B >= 1 && s.T >= 1 && s.KV >= 1 && s.H % s.KV == 0 && s.qh == s.DH && s.kh == s.DH &&
           s.qt == (long long)s.H * s.DH && s.kt == (long long)s.KV * s.DH && (long long)s.B * s.H * ((s.T + XT - 1) / XT) * 4 <= 0x7fffffff;
}
static int map_rows(CUtensorMap* m, const void* base, const AttnShape& s, int heads, int rows) {
    uint64_t dims[4] = {(uint64_t)s.DH, (uint64_t)heads, (uint64_t)s.T, (uint64_t)s.B};
    uint64_t strides[3] = {(uint64_t)s.DH * 2, (uint64_t)heads * s.DH * 2, (uint64_t)s.T * heads * s.DH * 2};
    uint32_t box[4] = {XD, 1, (uint32_t)rows, 1};
    return tc_make_tmap_bf16(m, base, 4, dims, strides, box, 128);
}
// Where the line to attn_mma.cu lies.  Its 64-row tiles and lower set-up win where 128-row tiles are half empty or the SMs are not full.
// Forward, us there / here (row after row of launches, heads = batch x heads): T64 384 heads 5.2 / 9.2, T20 960 heads 10.2 / 17.6, so up to 64
// rows never here; T100 296 heads 9.6 / 6.2 (cold 16.3 / 13.3, but 192 heads 12.4 / 12.4 and 96 heads 10.5 / 10.8), 384 heads 10.8 / 10.0;
// T129 64 heads 9.4 / 7.6, 148 heads 9.9 / 7.7, 168 heads 9.8 / 11.3, 225 heads 12.2 / 12.2, 256 heads 13.4 / 12.7, 300 heads 15.1 / 16.0, 608 heads
// 28.3 / 27.7: two of its tiles against three there, and a last wave of CTAs (two to an SM) that is less than half full tips it;
// T193 168 heads 14.4 / 11.2.
static bool forward_here(const AttnShape& s) {
    const long long ctas = (long long)s.B * s.H * ((s.T + XT - 1) / XT), wave = 2 * AX_SMS, last = ctas % wave;
    if (s.T <= 64) return false;
    if (s.T <= XT) return ctas > wave;
    return s.T > 192 || ctas <= wave || ctas > 4 * wave || last == 0 || last >= wave / 2;
}
// Backward, by its 128 x 64 steps (us there / here, row after row of launches).  Up to one step an SM never here: 48 (8 heads KV 4 T193) 18.7 / 22.7,
// 144 (24 heads KV 8 T256) 22.7 / 26.8.  Above, a CTA of dK / dV has to have something to walk for its 512 TMEM columns: a single step each never pays
// (kv heads as heads, up to 64 rows: 192 heads T20 12.4 / 18.6, 384 heads T64 18.5 / 27.7), two do while all of them are at work at
// once (144 heads T65 24.1 / 16.5 and 296 heads T65 26.0 / 24.7, but 608 heads T65 45.2 / 51.1 and 384 heads T129 53.4 / 59.5).  And up to
// two steps an SM the kernels there have SMs to spare as long as their 64-row tiles are few and the walks short: 8 heads KV 4 T500 28.8 / 30.9, 16
// heads KV 8 T384 26.9 / 28.8, but 16 heads KV 2 T384 43.1 / 37.0, 8 heads KV 8 T640 36.9 / 32.9, 64 heads T129 24.7 / 18.6 (just
// above the line 48 heads KV 16 T129 lose: 20.7 / 22.8).
static long long steps(const AttnShape& s) {
    const long long tiles = (s.T + XT - 1) / XT, nq = (s.T + XQ - 1) / XQ;
    return s.B * s.H * (tiles * nq - tiles * (tiles - 1));
}
static bool backward_here(const AttnShape& s) {
    const long long st = steps(s), nq = (s.T + XQ - 1) / XQ, key_tiles = (long long)s.B * s.KV * ((s.T + XT - 1) / XT);
    if (st <= AX_SMS || st <= key_tiles || (st <= 2 * key_tiles && key_tiles > 2 * AX_SMS)) return false;
    return st > 2 * AX_SMS || (long long)s.B * s.H * nq > 128 || s.H / s.KV * nq >= 20 || nq > 8;
}
// CTAs to a key tile in the dK / dV kernel.  The first key tile walks the steps of all query tiles of the group's heads, `chain` of them; an
// even share of all steps over the SMs is `share`.  Backward in us with S = 1 / 2 / 4 CTAs to a tile (chain / share): B2 H16 KV2 T900 (120 / 13)
// 173 / 110 / 79, B2 H8 KV2 T500 DH48 (32 / 2) 60 / 46 / 40, B1 H12 KV4 T2500 (120 / 34) 204 / 143 / 145, B1 H32 KV8 T1400 (88 / 28) 152 / 107 / 118,
// B4 H24 KV8 T500 (24 / 12) 65 / 67 / 96, B2 H4 KV2 T200 (8 / 0) 28 / 28 / 28; eight are no better anywhere.
// Clusters that do not all run at once (74 of two, 33 of four fit the GPU) start late: that is no loss only where the first tile's share of
// the walk outlasts all of it spread over those that run, with two steps for the set-up and the merge of each of four and one of each
// of two.  1 / 2 / 4 with that many key tiles: 36 (B3 H12 KV4 T384) 35 / 33 / 41, 40 (B1 H16 KV8 T640) 45 / 37 / 45, 72 (B1 H8 KV8 T1100) 51 / 45 / 66,
// 112 (B7 H24 KV8 T129) 31 / 38 / 58, but 40 (B1 H4 KV2 T2500) 139 / 105 / 85, 36 (B1 H8 KV4 T1100) 66 / 55 / 49, 128 (B2 H24 KV8 T900) 83 / 70 / 102.
static int parts(const AttnShape& s) {
    const long long nq = (s.T + XQ - 1) / XQ, chain = s.H / s.KV * nq, st = steps(s), share = st / AX_SMS, key_tiles = (long long)s.B * s.KV * ((s.T + XT - 1) / XT);
    auto fit = [&](int n, int at_once) { return key_tiles <= at_once || at_once * chain > st + n * n / 2 * key_tiles; };
    int S = 1;
    while (S < 4 && chain >= 8 * S && chain > 2 * S * share && fit(2 * S, S == 1 ? AX_SMS / 2 : 33)) S *= 2;
    return S;
}
int ax_attn_tcs_route(int backward, const AttnShape& s) {
    if (!served(s)) return 0;
    return backward ? (backward_here(s) ? parts(s) : 0) : forward_here(s);
}
int ax_attn_fwd_tcs(const void* q, const void* k, const void* v, void* o, float* lse, const AttnShape& s, int* status, cudaStream_t st) {
    if (!ax_attn_tcs_route(0, s) || !lse || !aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o)) return -1;
    CUtensorMap tq, tk, tv;
    if (map_rows(&tq, q, s, s.H, XT) || map_rows(&tk, k, s, s.KV, XT) || map_rows(&tv, v, s, s.KV, XT)) return 2;
    const dim3 grid((s.T + XT - 1) / XT * s.H * s.B);
    ax_variant = 0x80;
    return ax_launch_chain(k_attn_fwd_tcs, grid, dim3(XF_THREADS), XFwdSmem::TOTAL, st, tq, tk, tv, (bf16*)o, lse, s.T, s.H, s.KV, s.DH, s.scale, status) == cudaSuccess ? 0 : 3;
}
int ax_attn_bwd_tcs(const void* q, const void* k, const void* v, const void* dO, const float* lse, const float* Dv, void* dq, void* dk, void* dv,
                    const AttnShape& s, const float* rope_cos, const float* rope_sin, int* status, cudaStream_t st) {
    if (rope_cos && (s.DH != XD || !rope_sin || !aligned16(rope_cos) || !aligned16(rope_sin))) return -1;
    if (!ax_attn_tcs_route(1, s) || !lse || !aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(dO) || !aligned16(dq) || !aligned16(dk) || !aligned16(dv)) return -1;
    CUtensorMap q128, g128, k64, v64, q64, g64, k128, v128;
    if (map_rows(&q128, q, s, s.H, XT) || map_rows(&g128, dO, s, s.H, XT) || map_rows(&k64, k, s, s.KV, XQ) || map_rows(&v64, v, s, s.KV, XQ) ||
        map_rows(&q64, q, s, s.H, XQ) || map_rows(&g64, dO, s, s.H, XQ) || map_rows(&k128, k, s, s.KV, XT) || map_rows(&v128, v, s, s.KV, XT)) return 2;
    const int tiles = (s.T + XT - 1) / XT;
    if (ax_launch_chain(k_attn_dq_tcs, dim3(tiles * s.H * s.B), dim3(XG_THREADS), XdQSmem::TOTAL, st, q128, g128, k64, v64, lse, Dv, (bf16*)dq, s,
                        rope_cos, rope_sin, status) != cudaSuccess) return 3;
    const int S = parts(s);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles * s.KV * s.B * S); cfg.blockDim = dim3(XK_THREADS); cfg.dynamicSmemBytes = XdKVSmem::TOTAL; cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = ax_gemm_pdl() ? 2 : 1;
    ax_variant = 0x81;
    return cudaLaunchKernelEx(&cfg, k_attn_dkv_tcs, q64, g64, k128, v128, lse, Dv, (bf16*)dk, (bf16*)dv, s, S, rope_cos, rope_sin, status) == cudaSuccess ? 0 : 3;
}
