// The single-model form (M = 1) of the fused tensor-core E-step (estep_tc.cuh).
//
// With one model the responsibility v of a kept sample is 1, so nothing has to
// be known about the other channels before the statistics can be summed: the
// two phases of the general form (log-densities first, then, after the exchange
// of Lt between the models, everything again weighted by v) become one.  Per
// (sample, channel) the general form issues 5m MUFU operations, this one 3m + 2
// (lg2, ex2 for |y|^(rho-2), ex2 for the responsibility; one reciprocal and one
// lg2 for the log-sum-exp), no log2|y| goes through tensor memory and no
// log-sum-exp through shared memory.  What that frees holds
//   W_hi in tensor memory beside W_lo (both MMA1 halves take A from there), and
//   two sets of G and b operand tiles in shared memory instead of one, so that a
//   density warp that is done with a tile goes on to the next without waiting
//   for the slowest warp and the MMA2 that follows it.
// Lt(t) = P(t) is the channel sum of the log-sum-exp: each warp leaves its sum
// per sample in one of three shared-memory rows, and the first warp of a sample
// set adds the set's warps one tile later.
//
// Bound by the latency of the density warps' instructions (12 warps per SM; in
// the counters at n = 64, T = 500k, m = 3: 49% of issue slots, MUFU pipe 52% busy).
// E-step, general form -> this one: n = 32, T = 60k, m = 3: 37.0 -> 24.7 us; n = 64,
// T = 500k, m = 1 / 2 / 3: 136 / 187 / 244 -> 99 / 129 / 161 us; n = 64, T = 300k,
// m = 5: 259 (2 warpgroups) -> 168 us; n = 128, T = 400k, m = 3: 376 -> 242 us.
#pragma once
#include "estep_tc.cuh"

namespace {

template <class Cf>
struct OneShape {
    static constexpr int kS = Cf::kS;
    static constexpr int NST = Cf::kNST;
    static constexpr uint32_t X_BYTES = (uint32_t)kS * 128u * 4u;
    static constexpr uint32_t G_BYTES = 128u * 128u * ((kS + 31) / 32);
    static constexpr uint32_t OFF_X0 = 0;
    static constexpr uint32_t OFF_G = OFF_X0 + NST * X_BYTES;          // [2 sets][G, b]
    static constexpr uint32_t OFF_SLOT = OFF_G + 4 * G_BYTES;          // [3 tiles][4 warps][kS] channel sums
    static constexpr uint32_t OFF_BAR = OFF_SLOT + 3 * 4 * kS * 4;
    static constexpr uint32_t NBAR = 32;
    static constexpr uint32_t OFF_MISC = OFF_BAR + NBAR * 8;
    static constexpr uint32_t BYTES = OFF_MISC + 64;
    static_assert(BYTES + 1024 <= 232448, "shared memory");
    __device__ static constexpr uint32_t g_off(int set) { return OFF_G + (uint32_t)set * 2 * G_BYTES; }
};
// tensor memory: b [0, kS) and [64, 64 + kS); phi [128, 256); W_lo [256, 384); W_hi [384, 512)
constexpr int kOneWhiCol = 384;
enum { ONE_FULL0 = 0, ONE_EMPTY0 = kMaxStages, ONE_BFULL0 = 2 * kMaxStages, ONE_BEMPTY0 = ONE_BFULL0 + 2,
       ONE_GFULL0 = ONE_BEMPTY0 + 2, ONE_GEMPTY0 = ONE_GFULL0 + 2, ONE_PSI = ONE_GEMPTY0 + 2, ONE_DRAIN,
       ONE_LT0 /* 2 parities x 4 warpgroups */, ONE_NBAR = ONE_LT0 + 8 };

template <class Cf>
__device__ __forceinline__ void one_barriers(uint64_t* bar, bool reinit) {
    if (reinit)                                        // every wait on the previous item's has completed
        for (int r = 0; r < ONE_NBAR; r++)
            asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(&bar[r])) : "memory");
    for (int q = 0; q < kMaxStages; q++) {
        mbar_init(&bar[ONE_FULL0 + q], 1);
        mbar_init(&bar[ONE_EMPTY0 + q], 1);
    }
    for (int q = 0; q < 2; q++) {
        mbar_init(&bar[ONE_BFULL0 + q], 1);
        mbar_init(&bar[ONE_BEMPTY0 + q], Cf::kDensWarps);
        mbar_init(&bar[ONE_GFULL0 + q], Cf::kDensWarps);
        mbar_init(&bar[ONE_GEMPTY0 + q], 1);
    }
    mbar_init(&bar[ONE_PSI], 1);
    mbar_init(&bar[ONE_DRAIN], 1);
    for (int w = 0; w < 8; w++) mbar_init(&bar[ONE_LT0 + w], 4);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// W_hi = tf32(W) and W_lo = tf32(W - W_hi), block-diagonal diag(W, ..., W) of R
// blocks, into tensor memory (row -> lane): the density warps, the 16-column
// chunks dealt to the warpgroups.
template <class Cf>
__device__ __forceinline__ void one_load_w(const float* __restrict__ Wf, int npc, uint32_t tmem, int warp, int lane) {
    const int q4 = warp & 3, i = q4 * 32 + lane, si = i / npc;
    const float* Wrow = Wf + (size_t)(i - si * npc) * npc;
    const uint32_t la = tmem + ((uint32_t)(q4 * 32) << 16);
#pragma unroll 1
    for (int k0 = 16 * (warp >> 2); k0 < 128; k0 += 16 * Cf::kWG) {
        float hi[16], lo[16];
        const bool blk = (k0 / npc) == si;             // 16 columns never straddle a block
#pragma unroll
        for (int q = 0; q < 16; q += 4) {
            float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
            if (blk) w = *reinterpret_cast<const float4*>(Wrow + (k0 - si * npc + q));
            const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                hi[q + e] = tf32_rna(wv[e]);
                lo[q + e] = tf32_rna(wv[e] - hi[q + e]);
            }
        }
        tmem_st16(la + kOneWhiCol + (uint32_t)k0, hi);
        tmem_st16(la + kWloCol + (uint32_t)k0, lo);
    }
}

// The control thread's part of one item (tiles tile0 + k stride, k < ntl): x
// loads, MMA1(k) into b buffer k & 1, MMA2(k - 1) from operand set (k - 1) & 1.
template <class Cf>
__device__ __forceinline__ void one_control(uint8_t* sm, uint64_t* bar, volatile int* abort_flag, int* err,
                                            const CUtensorMap* map, uint32_t tmem, int64_t tile0, int64_t stride,
                                            int ntl) {
    using Sh = OneShape<Cf>;
    constexpr int kS = Cf::kS, NST = Sh::NST;
    const uint32_t sbase = smem_u32(sm);
    auto issue_tma = [&](int kt) {
        const int s = kt % NST;
        const int row = (int)((tile0 + (int64_t)kt * stride) * kS);
        mbar_expect_tx(&bar[ONE_FULL0 + s], Sh::X_BYTES);
#pragma unroll
        for (int cb = 0; cb < 4; cb++)
            tma_load_2d(sbase + Sh::OFF_X0 + (uint32_t)s * Sh::X_BYTES + (uint32_t)(cb * kS * 128), map, cb * 32, row,
                        &bar[ONE_FULL0 + s]);
    };
    constexpr uint32_t ID1 = idesc_tf32(128, kS, 0, 0);
    constexpr uint32_t ID2 = idesc_tf32(128, 128, 0, 0);
    auto mma2 = [&](int kp) {
        const uint32_t gb = sbase + Sh::g_off(kp & 1);
        const uint64_t ad0 = sdesc(gb, 16, 1024), bd0 = sdesc(gb + Sh::G_BYTES, 16, 1024);
#pragma unroll
        for (int kk = 0; kk < kS / 8; kk++) {
            const uint32_t off = (uint32_t)((kk >> 2) * 128 * 128 + (kk & 3) * 32) >> 4;
            tc_mma_tf32(tmem + kPsiCol, ad0 + off, bd0 + off, ID2, (kp > 0 || kk > 0) ? 1u : 0u);
        }
    };
    int issued = 0, consumed = 0;
    while (issued < NST && issued < ntl) issue_tma(issued++);
    bool ok = true;
    for (int k = 0; k < ntl && ok; k++) {
        const int s = k % NST, d = k & 1;
        ok = mbar_wait(&bar[ONE_FULL0 + s], (uint32_t)((k / NST) & 1), abort_flag, err);
        if (ok) consumed = k + 1;
        if (ok && k >= 2) ok = mbar_wait(&bar[ONE_BEMPTY0 + d], (uint32_t)(((k >> 1) - 1) & 1), abort_flag, err);
        if (!ok) break;
        tc_fence_after();
        const uint64_t bd0 = sdesc(sbase + Sh::OFF_X0 + (uint32_t)s * Sh::X_BYTES, 16, 1024);
        // the W_lo products first, then the W_hi ones on top (estep_tc.cuh)
#pragma unroll
        for (int kk = 0; kk < 16; kk++)
            tc_mma_tf32_ta(tmem + d * kBcol, tmem + kWloCol + (uint32_t)(kk * 8),
                           bd0 + (((uint32_t)((kk >> 2) * kS * 128 + (kk & 3) * 32)) >> 4), ID1, kk > 0 ? 1u : 0u);
#pragma unroll
        for (int kk = 0; kk < 16; kk++)
            tc_mma_tf32_ta(tmem + d * kBcol, tmem + kOneWhiCol + (uint32_t)(kk * 8),
                           bd0 + (((uint32_t)((kk >> 2) * kS * 128 + (kk & 3) * 32)) >> 4), ID1, 1u);
        tc_commit(&bar[ONE_EMPTY0 + s]);
        tc_commit(&bar[ONE_BFULL0 + d]);
        if (k >= 1) {
            const int kp = k - 1, gs = kp & 1;
            ok = mbar_wait(&bar[ONE_GFULL0 + gs], (uint32_t)((kp >> 1) & 1), abort_flag, err);
            if (!ok) break;
            tc_fence_after();
            mma2(kp);
            tc_commit(&bar[ONE_GEMPTY0 + gs]);
            // the stage that MMA1(k - 1) has read
            if (kp + NST < ntl) {
                ok = mbar_wait(&bar[ONE_EMPTY0 + kp % NST], (uint32_t)((kp / NST) & 1), abort_flag, err);
                if (!ok) break;
                issue_tma(kp + NST);
                issued = kp + NST + 1;
            }
        }
    }
    if (ok && ntl > 0) {
        const int kp = ntl - 1;
        ok = mbar_wait(&bar[ONE_GFULL0 + (kp & 1)], (uint32_t)((kp >> 1) & 1), abort_flag, err);
        if (ok) {
            tc_fence_after();
            mma2(kp);
            tc_commit(&bar[ONE_PSI]);
        }
    }
    // drain: every load issued has landed and every MMA has completed before the
    // CTA frees tensor memory or re-arms the barriers (bounded)
    for (int t = consumed; t < issued; t++)
        mbar_wait(&bar[ONE_FULL0 + (t % NST)], (uint32_t)((t / NST) & 1), abort_flag, err, false, false);
    tc_commit(&bar[ONE_DRAIN]);
    mbar_wait(&bar[ONE_DRAIN], 0u, abort_flag, err, false, false);
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
template <int MM>
__device__ __forceinline__ float2 max_pair(const float2* q) {
    float2 mx = q[0];
#pragma unroll
    for (int j = 1; j + 1 < MM; j += 2)
        mx = make_float2(max3(mx.x, q[j].x, q[j + 1].x), max3(mx.y, q[j].y, q[j + 1].y));
    if constexpr (MM % 2 == 0) mx = make_float2(fmaxf(mx.x, q[MM - 1].x), fmaxf(mx.y, q[MM - 1].y));
    return mx;
}

// The density warps' part of one item.  Arithmetic on pairs of consecutive
// samples (estep_tc.cuh): per mixture y, L2 = log2 max(|y|, kYFloor),
// q2 = 2^((rho-2) L2), p = q2 y^2 and q = log2 of its term; e_j = 2^(q_j - max),
// z_j = e_j / sum e; then the seven sums A0..A6 of tcp2 and g.
template <int MM, int R, class Cf>
__device__ __forceinline__ void one_density(uint8_t* sm, uint64_t* bar, volatile int* abort_flag, const EStepArgs& a,
                                            uint32_t tmem, int warp, int lane, int64_t tile0, int64_t stride,
                                            int ntl, int item_slot) {
    using Sh = OneShape<Cf>;
    constexpr int kS = Cf::kS, kWG = Cf::kWG, kSub = Cf::kSub;
    constexpr int npc = 128 / R, wps = npc / 32;       // channels and warps per sample set
    constexpr int kUnrollG4 = MM <= 3 ? kSub / 4 : 1;
    const int wg = warp >> 2, q4 = warp & 3;
    const int set = q4 / wps;
    const bool lead = (q4 % wps) == 0;
    const int tl = q4 * 32 + lane;
    const int n = a.n, ch = tl - set * npc;
    const bool ch_ok = ch < n;
    const uint32_t lane_addr = (uint32_t)(q4 * 32) << 16;
    float* slot = (float*)(sm + Sh::OFF_SLOT);
    MixT2 PS[MM];
#pragma unroll
    for (int j = 0; j < MM; j++) {
        const MixParam q = a.mp[(size_t)j * npc + ch];
        PS[j].s = f2s(q.s);
        PS[j].npo = f2s(-q.off);
        PS[j].pc = f2s(q.cl2);
        PS[j].pm2 = f2s(q.rho - 2.f);
        PS[j].sr = f2s(q.s * q.rho);
    }
    const float2 nwci2 = f2s(-a.wc[ch]);
    // padding channels have W = 0, s = 0: y, b and g are 0 there, and this
    // normaliser makes their log-sum-exp exactly 0 (lg2(m) - lg2(m))
    if (!ch_ok) {
#pragma unroll
        for (int j = 0; j < MM; j++) PS[j].pc = f2s(MM > 1 ? -ptx_lg2((float)MM) : 0.f);
    }
    float2 acc[MM][7];
    float2 fCn, fS2;
    auto zero_acc = [&]() {
#pragma unroll
        for (int j = 0; j < MM; j++)
#pragma unroll
            for (int k = 0; k < 7; k++) acc[j][k] = make_float2(0.f, 0.f);
        fCn = fS2 = make_float2(0.f, 0.f);
    };
    zero_acc();
    double dLL = 0.0, dVs = 0.0;
    PartLayout L{n, MM};
    double* out = a.partial + (size_t)((item_slot * R + set) * kWG + wg) * L.stride();
    double* out0 = a.partial + (size_t)((item_slot * R + set) * kWG) * L.stride();   // phi of this set
    // FP32 sums into this thread's entries of the slot: stored the first time, added after that
    bool first = true;
    auto flush = [&]() {
        if (ch_ok) {
            auto put = [&](double* p, double v) {
                if (first) *p = v;
                else red_add_f64(p, v);
            };
#pragma unroll
            for (int j = 0; j < MM; j++) {
                auto s = [&](int k) -> float { return acc[j][k].x + acc[j][k].y; };
                double us, kn, ln, mn, md, bd, rn;
                mix_stats_from_sums(s(0), s(1), s(2), s(3), s(4), s(5), s(6), PS[j].pm2.x + 2.f, a.grad_mode,
                                    a.update_rho, us, kn, ln, mn, md, bd, rn);
                const int o = j * n + ch;
                put(out + L.mix(kUs) + o, us);
                put(out + L.mix(kKn) + o, kn);
                put(out + L.mix(kLn) + o, ln);
                put(out + L.mix(kMn) + o, mn);
                put(out + L.mix(kMd) + o, md);
                put(out + L.mix(kBd) + o, bd);
                put(out + L.mix(kRn) + o, rn);
            }
            put(out + L.cn() + ch, (double)fCn.x + (double)fCn.y);
            put(out + L.s2() + ch, (double)fS2.x + (double)fS2.y);
            // (the slot's sum g serves the forms that sum g x^T; phi needs none)
        }
        first = false;
        zero_acc();
    };
    // lane t < kSub owns packed row t of this warpgroup's slice, sample (t0 + t) R + set
    const int lt = lane < kSub ? lane : kSub - 1;
    auto sample_of = [&](int k) -> int64_t {
        return ((tile0 + (int64_t)k * stride) * kS + wg * kSub + lt) * R + set;
    };
    auto keep_of = [&](int k) -> int {
        const int64_t t = sample_of(k);
        return k < ntl && t < a.T ? (a.keep != nullptr ? (int)a.keep[t] : 1) : 0;
    };
    // P(t) = Lt(t) of tile k (relative to the Lt constant), whose channel sums are in the slot row k % 3
    auto finish_p = [&](int k, uint32_t vmask) {
        if (lane < kSub) {
            const float* sq = slot + (k % 3) * 4 * kS + wg * kSub + lane;
            float sw = sq[set * wps * kS];
#pragma unroll
            for (int w = 1; w < wps; w++) sw += sq[(set * wps + w) * kS];
            const float P = kLn2 * sw;
            const int64_t t = sample_of(k);
            if ((vmask >> lane) & 1u) {
                dVs += 1.0;
                dLL += (double)P;
            }
            if (t < a.T) {
                if (a.Lt_out) a.Lt_out[t] = P;
                if (a.P_out) a.P_out[t] = P;
            }
        }
    };
    int keepv = keep_of(0);
    uint32_t vmask = 0;
    bool ok = true;
    for (int k = 0; k < ntl && ok; k++) {
        const int s = k & 1;
        const uint32_t u = (uint32_t)(k >> 1);
        const uint32_t vprev = vmask;
        vmask = __ballot_sync(0xffffffffu, lane < kSub && keepv != 0);
        keepv = keep_of(k + 1);                        // used one tile later
        ok = mbar_wait(&bar[ONE_BFULL0 + s], u & 1, abort_flag, a.err);
        // the operand set is free once MMA2 of tile k - 2 has run
        if (ok && k >= 2) ok = mbar_wait(&bar[ONE_GEMPTY0 + s], (u - 1) & 1, abort_flag, a.err);
        if (!ok) break;
        tc_fence_after();
        const uint32_t bcol = tmem + lane_addr + (uint32_t)(s * kBcol + wg * kSub);
        float* srow = slot + ((k % 3) * 4 + q4) * kS + wg * kSub;
        uint32_t bnext[4];
        tmem_ld4_nowait(bcol, bnext);
#pragma unroll kUnrollG4
        for (int g4 = 0; g4 < kSub / 4; g4++) {
            float v[4], gq[4], bq[4];
            tmem_wait_ld(bnext);
            const float2 b2[2] = {make_float2(__uint_as_float(bnext[0]), __uint_as_float(bnext[1])),
                                  make_float2(__uint_as_float(bnext[2]), __uint_as_float(bnext[3]))};
            if (g4 + 1 < kSub / 4) tmem_ld4_nowait(bcol + (uint32_t)(g4 * 4 + 4), bnext);
            float2 v2[2] = {f2s(1.f), f2s(1.f)};
            if (vmask != (1u << kSub) - 1u) {          // the same in every lane
                const uint32_t m4 = vmask >> (g4 * 4);
                v2[0] = make_float2((float)(m4 & 1u), (float)((m4 >> 1) & 1u));
                v2[1] = make_float2((float)((m4 >> 2) & 1u), (float)((m4 >> 3) & 1u));
            }
#pragma unroll
            for (int rp = 0; rp < 2; rp++) {
                const int r0 = 2 * rp, r1 = 2 * rp + 1;
                const float2 vv = v2[rp];
                float2 y[MM], L2[MM], q2[MM], p[MM], z[MM];
#pragma unroll
                for (int j = 0; j < MM; j++) {
                    y[j] = __ffma2_rn(PS[j].s, b2[rp], PS[j].npo);
                    L2[j] = make_float2(ptx_lg2(fmaxf(fabsf(y[j].x), kYFloor)), ptx_lg2(fmaxf(fabsf(y[j].y), kYFloor)));
                    const float2 e = __fmul2_rn(PS[j].pm2, L2[j]);
                    q2[j] = make_float2(ptx_ex2(e.x), ptx_ex2(e.y));
                    p[j] = __fmul2_rn(q2[j], __fmul2_rn(y[j], y[j]));
                    z[j] = __ffma2_rn(f2s(-kLog2e), p[j], PS[j].pc);
                }
                const float2 mx = max_pair<MM>(z);
                float2 lse = mx, rs = vv;
                if constexpr (MM > 1) {
                    float2 S;
#pragma unroll
                    for (int j = 0; j < MM; j++) {
                        const float2 d = __ffma2_rn(mx, f2s(-1.f), z[j]);
                        z[j] = make_float2(ptx_ex2(d.x), ptx_ex2(d.y));
                        S = j == 0 ? z[0] : __fadd2_rn(S, z[j]);
                    }
                    lse = __fadd2_rn(mx, make_float2(ptx_lg2(S.x), ptx_lg2(S.y)));
                    rs = __fmul2_rn(vv, make_float2(ptx_rcp(S.x), ptx_rcp(S.y)));
                } else {
                    z[0] = f2s(1.f);
                }
                v[r0] = lse.x;
                v[r1] = lse.y;
                float2 g = make_float2(0.f, 0.f);
#pragma unroll
                for (int j = 0; j < MM; j++) {
                    const float2 uu = __fmul2_rn(z[j], rs);
                    const float2 w = __fmul2_rn(uu, q2[j]);
                    const float2 gj = __fmul2_rn(w, y[j]);
                    const float2 wp = __fmul2_rn(uu, p[j]);
                    acc[j][0] = __fadd2_rn(acc[j][0], uu);
                    acc[j][1] = __fadd2_rn(acc[j][1], wp);
                    acc[j][2] = __ffma2_rn(wp, p[j], acc[j][2]);
                    acc[j][3] = __ffma2_rn(wp, L2[j], acc[j][3]);
                    acc[j][4] = __fadd2_rn(acc[j][4], gj);
                    acc[j][5] = __fadd2_rn(acc[j][5], w);
                    acc[j][6] = __ffma2_rn(wp, q2[j], acc[j][6]);
                    g = __ffma2_rn(PS[j].sr, gj, g);
                }
                const float2 bb = __fadd2_rn(b2[rp], nwci2);
                const float2 bv = __fmul2_rn(vv, bb);
                fCn = __fadd2_rn(fCn, bv);
                fS2 = __ffma2_rn(bv, bb, fS2);
                gq[r0] = tf32_half_up(g.x); gq[r1] = tf32_half_up(g.y);
                bq[r0] = tf32_half_up(bb.x); bq[r1] = tf32_half_up(bb.y);
            }
            const uint32_t goff = Sh::g_off(s) + sw128_off(tl, wg * kSub + g4 * 4, 128);
            *reinterpret_cast<float4*>(sm + goff) = make_float4(gq[0], gq[1], gq[2], gq[3]);
            *reinterpret_cast<float4*>(sm + goff + Sh::G_BYTES) = make_float4(bq[0], bq[1], bq[2], bq[3]);
            // channel sums: a 4-value transposed butterfly, lane 8q ends with sample 4 g4 + q
            {
                const bool up16 = (lane & 16) != 0;
                const float s0 = up16 ? v[0] : v[2], s1 = up16 ? v[1] : v[3];
                const float k0 = up16 ? v[2] : v[0], k1 = up16 ? v[3] : v[1];
                v[0] = k0 + __shfl_xor_sync(0xffffffffu, s0, 16);
                v[1] = k1 + __shfl_xor_sync(0xffffffffu, s1, 16);
                const bool up8 = (lane & 8) != 0;
                const float s2 = up8 ? v[0] : v[1], k2 = up8 ? v[1] : v[0];
                float w = k2 + __shfl_xor_sync(0xffffffffu, s2, 8);
                w += __shfl_xor_sync(0xffffffffu, w, 4);
                w += __shfl_xor_sync(0xffffffffu, w, 2);
                w += __shfl_xor_sync(0xffffffffu, w, 1);
                if ((lane & 7) == 0) srow[g4 * 4 + ((lane >> 4) & 1) * 2 + ((lane >> 3) & 1)] = w;
            }
        }
        // operand set s written, b buffer s consumed
        fence_proxy_async();
        tc_fence_before();
        __syncwarp();
        if constexpr (wps == 1) {
            finish_p(k, vmask);
        } else if (k >= 1 && lead) {
            ok = mbar_wait(&bar[ONE_LT0 + (s ^ 1) * 4 + wg], (uint32_t)(((k - 1) >> 1) & 1), abort_flag, a.err);
            if (ok) finish_p(k - 1, vprev);
            __syncwarp();
        }
        if (lane == 0) {
            // in this order: MMA1(k + 2) waits for every warp's arrival at BEMPTY,
            // so by then each has arrived at this tile's Lt barrier (which tile
            // k + 2 uses again) and the lead warps have read the slot row of tile
            // k - 1 (which tile k + 2 writes)
            if constexpr (wps > 1) mbar_arrive(&bar[ONE_LT0 + s * 4 + wg]);
            mbar_arrive(&bar[ONE_BEMPTY0 + s]);
            mbar_arrive(&bar[ONE_GFULL0 + s]);
        }
        if ((k + 1) % kFlush == 0) flush();
    }
    if (wps > 1 && ok && ntl > 0 && lead) {
        ok = mbar_wait(&bar[ONE_LT0 + ((ntl - 1) & 1) * 4 + wg], (uint32_t)(((ntl - 1) >> 1) & 1), abort_flag, a.err);
        if (ok) finish_p(ntl - 1, vmask);
    }
    if (first || ntl % kFlush != 0) flush();
    if (lead) {
        double a1 = dLL, a2 = dVs;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a1 += __shfl_xor_sync(0xffffffffu, a1, o);
            a2 += __shfl_xor_sync(0xffffffffu, a2, o);
        }
        if (lane == 0) {
            out[0] = a1;
            out[1] = a2;
        }
    }
    // phi out of tensor memory: the diagonal block of this set, in 16-column
    // chunks dealt to the warpgroups
    if (ok && ntl > 0) ok = mbar_wait(&bar[ONE_PSI], 0u, abort_flag, a.err);
    if (ok && ntl > 0) {
        tc_fence_after();
#pragma unroll
        for (int c0 = 0; c0 < npc; c0 += 16) {
            if ((c0 / 16) % kWG != wg) continue;
            float v[16];
            tmem_ld16(tmem + kPsiCol + lane_addr + (uint32_t)(set * npc + c0), v);
#pragma unroll
            for (int q = 0; q < 16; q++)
                if (ch_ok && c0 + q < n) out0[L.psi() + (size_t)(c0 + q) * n + ch] = (double)v[q];
        }
    }
}

}  // namespace
