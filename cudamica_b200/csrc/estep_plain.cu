// Plain FP32 form of the fused AMICA E-step (SIMT FP32 contractions).
//
// One thread-block cluster per sample tile stream; CTA rank h of the cluster
// owns model h (cluster size = M).  Per tile of S samples each CTA:
//   1. stages the x tile in shared memory and computes b = W_h x on the FP32
//      pipe (register-blocked SIMT GEMM, W_h resident in shared memory);
//   2. evaluates the generalized-Gaussian mixture log-densities and the
//      log-sum-exp over mixtures per (channel, sample) -- the work of
//      betabyxminusmu / logalogblogpfun / updateltz (src/kernels.cu:251-366);
//   3. reduces over channels to Lt_h(t) and exchanges Lt over distributed
//      shared memory so that every CTA forms P(t) and v_h(t) (updatell,
//      src/kernels.cu:376-450) without touching global memory;
//   4. accumulates the sufficient statistics of src/kernels.cu:473-827 in
//      registers and Psi_h += g x^T (the sum behind phi = g b^T of
//      src/amica.cu:1535-1550, with phi formed from Psi in the FP64 M-step).
// Partial sums go to a per-CTA slot of `partial`; a separate kernel reduces
// the slots in a fixed order, so results are deterministic.
//
// Bound by the FP32 pipe and shared-memory loads of the two products and by MUFU
// latency with 8 to 12 warps per SM.  E-step in the middle of a fit, with lanes for 32,
// 64 or 128 channels, K always the padded count and runs of consecutive samples ->
// now: n = 71, T = 200k, M = 2, m = 3: 1039 -> 617 us; n = 128, T = 300k, M = 3: 2.52 -> 2.33
// ms; n = 256, T = 50k, M = 2, m = 5: 1.27 -> 1.19 ms; n = 100, T = 200k, M = 1: 565 -> 529 us;
// n = 32, T = 300k, M = 1: 199 -> 189 us.  At the start of a fit, where no responsibility is
// 0 yet: 1077 -> 652 us, 2.61 -> 2.57 ms, 1.27 -> 1.23 ms.
#include <cooperative_groups.h>
#include <cstdio>

#include <algorithm>

#include "common.cuh"
#include "density.cuh"

namespace cg = cooperative_groups;
using namespace amica;

namespace {

constexpr int kS = 64;  // samples per tile
// A tile's samples are four consecutive ones from each of 16 segments of the data
// (sample t of tile: segment t / 4): the models of consecutive samples are mostly
// the same, and a model skips the second phase of samples it has no
// responsibility for, so that with a run of samples one CTA of the cluster works
// while the others wait.
__device__ __forceinline__ int64_t plain_sample(int64_t tile, int t, int64_t ntiles) {
    return (int64_t)(t >> 2) * 4 * ntiles + 4 * tile + (t & 3);
}

// NP: channels as laid out (32, 64, 128 or 256); NA: channels worked on (96 for
// 65 to 96 of 128).  Up to 128 channels one CTA per model holds them all; at 256
// the Q = 4 CTAs of a model each own NPL = 64 channels (their rows of W, their
// densities, their rows of Psi) and read the full x tile; their per-sample channel
// sums are added in the cluster.
// 8 warps, 12 with NA = 96.  (16 warps at NA = 128 and 256, with half the register
// block each, are bound by shared-memory loads in the products: 2.47 against 2.36
// ms at n = 128, T = 300k, M = 3, and 1.58 against 1.26 at n = 256, T = 50k, M = 2.)
template <int NP, int NA, int MM>
struct PlainShape {
    static constexpr int NPL = NP <= 128 ? NA : 64; // channels of this CTA
    static constexpr int Q = NP <= 128 ? 1 : NP / NPL;   // CTAs per model
    static constexpr int THREADS = NPL == 96 ? 384 : 256;
    static constexpr int SPLIT = THREADS / NPL;     // sample groups per channel
    static constexpr int SUB = kS / SPLIT;          // samples per thread per tile
    static constexpr int NK = NP <= 128 ? NA : NP;  // columns of W and x held
    static constexpr int WLD = NPL + 4;             // padded row of W^T in smem
    static constexpr int XLD = NK + 4;              // padded row of the x tile
    // x tile: XROWS samples at a time, XUNROLL of a thread's loads in flight: all, but
    // with 2 to 4 mixtures at 128 channels, where the registers are short (m = 3: 322 us
    // against 330 at T = 60k, M = 2; m = 5 388 against 380, m = 1, M = 1 158 against 154).
    // One address from scratch per load cost 2 to 6% of the E-step.
    static constexpr int XROWS = THREADS / (NK / 4);
    static_assert(THREADS % (NK / 4) == 0 && XROWS % 4 == 0 && kS % XROWS == 0, "x tile");
    static constexpr int XUNROLL = NK == 128 && MM >= 2 && MM <= 4 ? 4 : kS / XROWS;
    // GEMM b = W x: each thread 4 channels x CT samples
    static constexpr int NTI = NPL / 4;
    static constexpr int NTT = THREADS / NTI;
    static constexpr int CT = kS / NTT;
    static_assert(NTI * NTT == THREADS && NTT * CT == kS, "b = W x tiling");
    // Psi update: each thread RI x RK block, RI in two runs of RL = RI / 2 channels (one
    // of two at NPL = 32, an 8-byte load: 205 -> 197 us at n = 32, T = 300k, M = 1, m = 3)
    static constexpr int RI = NPL / 16;
    static constexpr int RL = RI > 2 ? RI / 2 : RI;
    static constexpr int RK = NK / (THREADS / 16);
    static_assert(RK * (THREADS / 16) == NK && RI % 2 == 0, "Psi tiling");
    static constexpr int LLD = NPL + 8;             // padded row of the lse tile (8 lanes per sample)
    static constexpr int NACC = 7 * MM + 3;
    static constexpr size_t tile_floats = (size_t)kS * (XLD + NPL + NPL + LLD);
    // FP64 running sums: with 256 threads each keeps those of its own channel and
    // sample group in registers; with more the groups' FP32 sums are folded through
    // shared memory (the tile's place) into FP64 sums spread over the threads
    static constexpr bool REG64 = THREADS == 256;
    static constexpr size_t fold_floats = (size_t)NACC * THREADS * (REG64 ? 2 : 1);
    static constexpr size_t work_floats = tile_floats > fold_floats ? tile_floats : fold_floats;
    static constexpr size_t smem_floats = (size_t)NK * WLD + work_floats + 2 * kS + kS;
    static constexpr int NFOLD = REG64 ? NACC : (NACC * NPL + THREADS - 1) / THREADS;   // FP64 sums per thread
    // CTAs per SM: one mixture of up to 32 channels fits two into the registers (128 a
    // thread; 140 and one CTA: 169 us instead of 105 at n = 32, T = 300k, M = 1)
    static constexpr int CTAS = NPL == 32 && MM == 1 ? 2 : 1;
};

template <int NP, int NA, int MM>
__global__ void __launch_bounds__(PlainShape<NP, NA, MM>::THREADS, PlainShape<NP, NA, MM>::CTAS) estep_plain_kernel(EStepArgs a) {
    using Sh = PlainShape<NP, NA, MM>;
    constexpr int NPL = Sh::NPL, Q = Sh::Q, THREADS = Sh::THREADS, NK = Sh::NK, NACC = Sh::NACC;
    extern __shared__ __align__(16) float sm[];
    float* Wt = sm;                                   // [NK][WLD]  Wt[k][i] = W[i0 + i][k]
    float* xs = Wt + NK * Sh::WLD;                    // [S][XLD]
    float* bs = xs + kS * Sh::XLD;                    // [S][NPL]   (W x)_i per sample
    float* gs = bs + kS * NPL;                        // [S][NPL]   g
    float* lse = gs + kS * NPL;                       // [S][LLD]   log-sum-exp over mixtures
    float* slot = Wt + NK * Sh::WLD + Sh::work_floats;   // [2][S]  cluster-visible L_h(t)
    float* vS = slot + 2 * kS;                        // [S]        v_h(t) (0 if not used)

    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int h = rank / Q, cq = rank % Q;            // model, channel block
    const int i0c = cq * NPL;                         // first channel of this CTA
    const int cid = blockIdx.x / (a.M * Q);
    const int tid = threadIdx.x;
    const int n = a.n, M = a.M;
    if (a.m != MM || n > NP || (NP <= 128 && n > NA)) {
        if (tid == 0) atomicOr(a.err, kErrShape);
    }

    // ---- resident per-CTA data: W_h^T and this thread's mixture constants
    {
        const float* Wh = a.Wf + ((size_t)h * NP + i0c) * NP;
        for (int e = tid; e < NPL * NK; e += THREADS) {
            int i = e / NK, k = e % NK;
            Wt[k * Sh::WLD + i] = Wh[(size_t)i * NP + k];
        }
    }
    const int ch = tid % NPL;           // density-phase channel (of this CTA)
    const int grp = tid / NPL;          // density-phase sample group
    const int gch = i0c + ch;           // the channel's index in the model
    const bool ch_ok = gch < n;
    // mixtures (0,1), (2,3) as float2 pairs, an odd last one as a scalar
    constexpr int NPR = MM / 2;
    constexpr bool kOdd = (MM & 1) != 0;
    constexpr int NPRA = NPR > 0 ? NPR : 1;
    MixV<float2> P2[NPRA];
    MixV<float> P1;
#pragma unroll
    for (int j = 0; j < MM; j++) {
        const MixParam q = a.mp[((size_t)h * MM + j) * NP + gch];
        if (j < 2 * NPR) {
            float2* f[5] = {&P2[j / 2].s, &P2[j / 2].npo, &P2[j / 2].pc, &P2[j / 2].pr, &P2[j / 2].sr};
            const float vals[5] = {q.s, -q.off, q.cl2, q.rho, q.s * q.rho};
#pragma unroll
            for (int e = 0; e < 5; e++) {
                if (j & 1) f[e]->y = vals[e];
                else f[e]->x = vals[e];
            }
        } else {
            P1.s = q.s; P1.npo = -q.off; P1.pc = q.cl2; P1.pr = q.rho; P1.sr = q.s * q.rho;
        }
    }
    const float wci = a.wc[(size_t)h * NP + gch];
    // this model's offset of Lt; with Q > 1 the per-sample threads add every model's
    const float ltch = (float)(a.ltc64[h] - a.ltc64[0]);
    __shared__ float ltcs[kMaxModels];
    if (Q > 1 && tid < M) ltcs[tid] = (float)(a.ltc64[tid] - a.ltc64[0]);

    // FP32 sums of this thread's channel and sample group: A0..A6 of dens_acc per
    // mixture, sum v b, sum v b^2, sum g
    float2 fP[NPRA][7];
    float fS1[7], fCn, fS2, fGs;
    auto zero_sums = [&]() {
#pragma unroll
        for (int k = 0; k < 7; k++) {
#pragma unroll
            for (int qq = 0; qq < NPRA; qq++) fP[qq][k] = make_float2(0.f, 0.f);
            fS1[k] = 0.f;
        }
        fCn = fS2 = fGs = 0.f;
    };
    zero_sums();
    // FP64 running sums: REG64, this thread's NACC; else thread e owns the (sum, channel)
    // pairs e, e + THREADS, ... of NACC x NPL, the groups added in order
    double dF[Sh::NFOLD];
#pragma unroll
    for (int u = 0; u < Sh::NFOLD; u++) dF[u] = 0.0;
    auto fold = [&]() {                               // not REG64: between two barriers
        if constexpr (Sh::REG64) {
#pragma unroll
            for (int k = 0; k < 7; k++) {
#pragma unroll
                for (int qq = 0; qq < NPR; qq++) {
                    dF[k * MM + 2 * qq] += fP[qq][k].x;
                    dF[k * MM + 2 * qq + 1] += fP[qq][k].y;
                }
                if constexpr (kOdd) dF[k * MM + MM - 1] += fS1[k];
            }
            dF[7 * MM + 0] += fCn;
            dF[7 * MM + 1] += fS2;
            dF[7 * MM + 2] += fGs;
            zero_sums();
            return;
        }
        float* fb = xs;
#pragma unroll
        for (int k = 0; k < 7; k++) {
#pragma unroll
            for (int qq = 0; qq < NPR; qq++) {
                fb[(k * MM + 2 * qq) * THREADS + tid] = fP[qq][k].x;
                fb[(k * MM + 2 * qq + 1) * THREADS + tid] = fP[qq][k].y;
            }
            if constexpr (kOdd) fb[(k * MM + MM - 1) * THREADS + tid] = fS1[k];
        }
        fb[(7 * MM + 0) * THREADS + tid] = fCn;
        fb[(7 * MM + 1) * THREADS + tid] = fS2;
        fb[(7 * MM + 2) * THREADS + tid] = fGs;
        __syncthreads();
#pragma unroll
        for (int u = 0; u < Sh::NFOLD; u++) {
            const int e = tid + u * THREADS;
            if (e < NACC * NPL) {
                const int k = e / NPL, c = e - k * NPL;
#pragma unroll
                for (int g = 0; g < Sh::SPLIT; g++) dF[u] += (double)fb[k * THREADS + g * NPL + c];
            }
        }
        zero_sums();
    };
    double dLL = 0.0, dVs = 0.0;   // per-sample threads (tid < S)
    constexpr int PRI = Sh::RI, PRL = Sh::RL, PRK = Sh::RK;
    float psi[PRI][PRK];
#pragma unroll
    for (int r = 0; r < PRI; r++)
#pragma unroll
        for (int c = 0; c < PRK; c++) psi[r][c] = 0.f;
    const int kend = NK < ((n + 3) & ~3) ? NK : ((n + 3) & ~3);   // W and x are zero beyond n

    int it = 0;
    for (int tile = cid; tile < a.ntiles; tile += a.nclusters, it++) {
        const int par = it & 1;
        __syncthreads();                              // the last tile's (or fold's) readers are done
        // ---- stage the x tile (float4, coalesced; samples past T are zero): a thread's
        // samples are whole segments apart, so its pointer walks
        {
            const int tr = tid / (NK / 4), k4 = tid % (NK / 4);
            int64_t ts = plain_sample(tile, tr, a.ntiles);
            const int64_t dts = (int64_t)Sh::XROWS * a.ntiles, dxp = dts * a.ldx;
            const float* xp = a.x + ts * a.ldx + 4 * k4;
            float* xd = xs + tr * Sh::XLD + 4 * k4;
#pragma unroll(Sh::XUNROLL)
            for (int u = 0; u < kS / Sh::XROWS; u++) {
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (ts < a.T) v = *reinterpret_cast<const float4*>(xp);
                *reinterpret_cast<float4*>(xd) = v;
                ts += dts;
                xp += dxp;
                xd += Sh::XROWS * Sh::XLD;
            }
        }
        __syncthreads();
        // ---- b = W_h x  (thread: channels 4*ti..+3, samples tt*CT..+CT-1)
        {
            const int ti = tid % Sh::NTI, tt = tid / Sh::NTI;
            float acc[Sh::CT][4];
#pragma unroll
            for (int c = 0; c < Sh::CT; c++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[c][q] = 0.f;
#pragma unroll 2
            for (int k = 0; k < kend; k += 4) {
                float4 w0 = *reinterpret_cast<const float4*>(Wt + (k + 0) * Sh::WLD + 4 * ti);
                float4 w1 = *reinterpret_cast<const float4*>(Wt + (k + 1) * Sh::WLD + 4 * ti);
                float4 w2 = *reinterpret_cast<const float4*>(Wt + (k + 2) * Sh::WLD + 4 * ti);
                float4 w3 = *reinterpret_cast<const float4*>(Wt + (k + 3) * Sh::WLD + 4 * ti);
#pragma unroll
                for (int c = 0; c < Sh::CT; c++) {
                    float4 xv = *reinterpret_cast<const float4*>(xs + (tt * Sh::CT + c) * Sh::XLD + k);
                    acc[c][0] = fmaf(w0.x, xv.x, acc[c][0]); acc[c][1] = fmaf(w0.y, xv.x, acc[c][1]);
                    acc[c][2] = fmaf(w0.z, xv.x, acc[c][2]); acc[c][3] = fmaf(w0.w, xv.x, acc[c][3]);
                    acc[c][0] = fmaf(w1.x, xv.y, acc[c][0]); acc[c][1] = fmaf(w1.y, xv.y, acc[c][1]);
                    acc[c][2] = fmaf(w1.z, xv.y, acc[c][2]); acc[c][3] = fmaf(w1.w, xv.y, acc[c][3]);
                    acc[c][0] = fmaf(w2.x, xv.z, acc[c][0]); acc[c][1] = fmaf(w2.y, xv.z, acc[c][1]);
                    acc[c][2] = fmaf(w2.z, xv.z, acc[c][2]); acc[c][3] = fmaf(w2.w, xv.z, acc[c][3]);
                    acc[c][0] = fmaf(w3.x, xv.w, acc[c][0]); acc[c][1] = fmaf(w3.y, xv.w, acc[c][1]);
                    acc[c][2] = fmaf(w3.z, xv.w, acc[c][2]); acc[c][3] = fmaf(w3.w, xv.w, acc[c][3]);
                }
            }
#pragma unroll
            for (int c = 0; c < Sh::CT; c++)
                *reinterpret_cast<float4*>(bs + (tt * Sh::CT + c) * NPL + 4 * ti) =
                    make_float4(acc[c][0], acc[c][1], acc[c][2], acc[c][3]);
        }
        __syncthreads();
        // ---- phase 1: per (channel, sample) log-sum-exp over mixtures (log2 units)
#pragma unroll 4
        for (int r = 0; r < Sh::SUB; r++) {
            const int t = grp * Sh::SUB + r;
            const float bx = bs[t * NPL + ch];
            float q[MM];
#pragma unroll
            for (int qq = 0; qq < NPR; qq++) {
                float2 L2;
                const float2 q2 = dens_q(P2[qq], bx, L2);
                q[2 * qq] = q2.x; q[2 * qq + 1] = q2.y;
            }
            if constexpr (kOdd) {
                float L2;
                q[MM - 1] = dens_q(P1, bx, L2);
            }
            lse[t * Sh::LLD + ch] = ch_ok ? lse2<MM>(q) : 0.f;
        }
        __syncthreads();
        // ---- Lt_h(t): the channel sum by 8 lanes per sample in a fixed
        // order, published for the cluster (with Q > 1, this CTA's channels only; the
        // blocks are added below)
        float* myslot = slot + par * kS;
        if (tid < 256) {                              // two rounds of 32 samples
#pragma unroll
            for (int t0r = 0; t0r < kS; t0r += 32) {
                const int t = t0r + (tid >> 3), j = tid & 7;
                float s = 0.f;
#pragma unroll
                for (int i = 0; i < NPL / 8; i++) s += lse[t * Sh::LLD + 8 * i + j];
                s += __shfl_xor_sync(0xffffffffu, s, 4);
                s += __shfl_xor_sync(0xffffffffu, s, 2);
                s += __shfl_xor_sync(0xffffffffu, s, 1);
                if (j == 0) myslot[t] = Q == 1 ? ltch + kLn2 * s : s;
            }
        }
        cluster.sync();
        // ---- P(t) and v_h(t) (identical arithmetic in every CTA of the cluster)
        if (tid < kS) {
            float L[kMaxModels];
            float lmax = -INFINITY;
#pragma unroll
            for (int q = 0; q < kMaxModels; q++) {
                if (q < M) {
                    if constexpr (Q == 1) {
                        const float* ps_q = cluster.map_shared_rank(myslot, q);
                        L[q] = ps_q[tid];
                    } else {
                        float s = 0.f;
#pragma unroll
                        for (int b = 0; b < Q; b++) s += cluster.map_shared_rank(myslot, q * Q + b)[tid];
                        L[q] = ltcs[q] + kLn2 * s;
                    }
                    lmax = fmaxf(lmax, L[q]);
                }
            }
            float se = 0.f, Lh = 0.f;
#pragma unroll
            for (int q = 0; q < kMaxModels; q++)
                if (q < M) {
                    se += ptx_ex2((L[q] - lmax) * kLog2e);
                    if (q == h) Lh = L[q];
                }
            const float P = lmax + kLn2 * ptx_lg2(se);
            const float vh = ptx_ex2((Lh - P) * kLog2e);
            const int64_t tg = plain_sample(tile, tid, a.ntiles);
            const bool valid = tg < a.T && (a.keep == nullptr || a.keep[tg]);
            vS[tid] = valid ? vh : 0.f;
            if (valid && cq == 0) {
                dVs += (double)vh;
                if (h == 0) dLL += (double)P;
            }
            if (tg < a.T && cq == 0) {
                if (a.Lt_out) a.Lt_out[(size_t)h * a.T + tg] = Lh;
                if (a.P_out && h == 0) a.P_out[tg] = P;
            }
        }
        __syncthreads();
        // ---- phase 2: responsibilities, score function and sufficient statistics
        {
            // the densities, responsibilities and sums of tile sample t; returns g
            auto sample = [&](int t) -> float {
                const float v = vS[t];
                // a sample whose model responsibility is exactly 0 adds exactly 0
                // to every sum and to g (v is the same in every lane of the warp)
                if (v == 0.f) return 0.f;
                const float bx = bs[t * NPL + ch];
                const float nl = -lse[t * Sh::LLD + ch];
                float2 g2 = make_float2(0.f, 0.f);
                float g1 = 0.f;
#pragma unroll
                for (int qq = 0; qq < NPR; qq++)
                    dens_acc<float2, false>(P2[qq], bx, make_float2(0.f, 0.f), nl, v, fP[qq], g2);
                if constexpr (kOdd) dens_acc<float, false>(P1, bx, 0.f, nl, v, fS1, g1);
                const float g = (g2.x + g2.y) + g1;
                const float bb = bx - wci;
                fCn = fmaf(v, bb, fCn);          // sum v b; cnew = A sum(v b) / vsum + c
                fS2 = fmaf(v * bb, bb, fS2);
                fGs += ch_ok ? g : 0.f;
                return g;
            };
#pragma unroll 2
            for (int r = 0; r < Sh::SUB; r++) {
                const int t = grp * Sh::SUB + r;
                const float g = sample(t);
                gs[t * NPL + ch] = ch_ok ? g : 0.f;
            }
        }
        if constexpr (Sh::REG64) fold();
        __syncthreads();
        // ---- Psi_h += g x^T over the tile (thread: RI x RK block, its channels in runs
        // NPL / 2 apart, so that a warp's loads of g are free of bank conflicts)
        {
            const int pi = tid % 16, pk = tid / 16;
            const int i0 = pi * PRL, k0 = pk * PRK;
            if (k0 < kend) {
#pragma unroll 4
                for (int t = 0; t < kS; t++) {
                    float gv[PRI], xv[PRK];
#pragma unroll
                    for (int r = 0; r < PRI; r++) gv[r] = gs[t * NPL + (r >= PRL ? NPL / 2 - PRL : 0) + i0 + r];
#pragma unroll
                    for (int c = 0; c < PRK; c++) xv[c] = xs[t * Sh::XLD + k0 + c];
#pragma unroll
                    for (int r = 0; r < PRI; r++)
#pragma unroll
                        for (int c = 0; c < PRK; c++) psi[r][c] = fmaf(gv[r], xv[c], psi[r][c]);
                }
            }
        }
        // FP32 sums cover at most 32 samples of a thread before they go to FP64
        if (!Sh::REG64 && par == 1) {
            __syncthreads();
            fold();
        }
    }
    __syncthreads();
    if constexpr (!Sh::REG64) fold();

    // ---- write this CTA's partial sums
    PartLayout L{n, MM};
    // one slot per (cluster, channel block); entries of the other blocks stay zero
    double* out = a.partial + ((size_t)(cid * Q + cq) * M + h) * L.stride();
    // the FP64 sums of a channel side by side, then mapped to the statistics
    double* red = reinterpret_cast<double*>(xs);      // [NACC][NPL]
    static_assert((size_t)NACC * NPL * 2 <= Sh::work_floats, "final sums");
    __syncthreads();
    if constexpr (Sh::REG64) {
#pragma unroll
        for (int k = 0; k < NACC; k++) red[k * THREADS + tid] = dF[k];
        __syncthreads();
        double s[(NACC * NPL + THREADS - 1) / THREADS];   // the groups added in order
#pragma unroll
        for (int u = 0; u * THREADS < NACC * NPL; u++) {
            const int e = tid + u * THREADS;
            s[u] = 0.0;
            if (e < NACC * NPL)
#pragma unroll
                for (int g = 0; g < Sh::SPLIT; g++) s[u] += red[(e / NPL) * THREADS + g * NPL + e % NPL];
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u * THREADS < NACC * NPL; u++)
            if (tid + u * THREADS < NACC * NPL) red[tid + u * THREADS] = s[u];
    } else {
#pragma unroll
        for (int u = 0; u < Sh::NFOLD; u++) {
            const int e = tid + u * THREADS;
            if (e < NACC * NPL) red[e] = dF[u];
        }
    }
    __syncthreads();
    for (int e = tid; e < MM * NPL; e += THREADS) {
        const int j = e / NPL, c = e - j * NPL, gi = i0c + c;
        if (gi >= n) continue;
        const float rho = a.mp[((size_t)h * MM + j) * NP + gi].rho;
        auto A = [&](int k) { return red[(k * MM + j) * NPL + c]; };
        double v[7];
        mix_stats_from_sums(A(0), A(1), A(2), A(3), A(4), A(5), A(6), rho, a.grad_mode, a.update_rho, v[kUs],
                            v[kKn], v[kLn], v[kMn], v[kMd], v[kBd], v[kRn]);
#pragma unroll
        for (int k = 0; k < 7; k++) out[L.mix(k) + j * n + gi] = v[k];
    }
    for (int c = tid; c < NPL; c += THREADS) {
        const int gi = i0c + c;
        if (gi >= n) continue;
        out[L.cn() + gi] = red[(7 * MM + 0) * NPL + c];
        out[L.s2() + gi] = red[(7 * MM + 1) * NPL + c];
        out[L.gs() + gi] = red[(7 * MM + 2) * NPL + c];
    }
    // LL numerator and vsum: per-sample threads, combined in fixed order
    __syncthreads();
    if (tid < kS) { red[tid] = dLL; red[kS + tid] = dVs; }
    __syncthreads();
    if (tid == 0 && cq == 0) {
        double s0 = 0.0, s1 = 0.0;
        for (int t = 0; t < kS; t++) { s0 += red[t]; s1 += red[kS + t]; }
        out[0] = s0;
        out[1] = s1;
    }
    {
        const int pi = tid % 16, pk = tid / 16;
        const int i0 = pi * PRL, k0 = pk * PRK;
#pragma unroll
        for (int r = 0; r < PRI; r++)
#pragma unroll
            for (int c = 0; c < PRK; c++) {
                const int i = i0c + (r >= PRL ? NPL / 2 - PRL : 0) + i0 + r, k = k0 + c;
                if (i < n && k < n) out[L.psi() + (size_t)k * n + i] = (double)psi[r][c];
            }
    }
    // peers may still read this CTA's slots: leave together
    cluster.sync();
}

// The launch of a shape, ready but for its grid.
template <int NP, int NA, int MM>
cudaError_t plain_config(int M, int nclusters, cudaStream_t st, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr) {
    using Sh = PlainShape<NP, NA, MM>;
    auto kern = estep_plain_kernel<NP, NA, MM>;
    const size_t smem = Sh::smem_floats * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int csize = M * Sh::Q;
    if (csize > 8) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
    }
    cfg = {};
    cfg.gridDim = dim3(nclusters * csize);
    cfg.blockDim = dim3(Sh::THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = csize;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaSuccess;
}

template <int NP, int NA, int MM>
cudaError_t launch_plain(const EStepArgs& a, int nclusters, cudaStream_t st) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    const cudaError_t e = plain_config<NP, NA, MM>(a.M, nclusters, st, cfg, attr);
    if (e != cudaSuccess) return e;
    return cudaLaunchKernelEx(&cfg, estep_plain_kernel<NP, NA, MM>, a);
}

// Largest cluster count whose clusters can all be resident at once (the grid
// is persistent: every cluster loops over its share of the tiles).
template <int NP, int NA, int MM>
int max_active_clusters(int M) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    if (plain_config<NP, NA, MM>(M, 64, nullptr, cfg, attr) != cudaSuccess) return -1;
    int num = 0;
    if (cudaOccupancyMaxActiveClusters(&num, estep_plain_kernel<NP, NA, MM>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    return num;
}

// channels worked on: 65 to 96 of 128 take three quarters of the lanes
int plain_work_channels(int n) { return n <= 32 ? 32 : n <= 64 ? 64 : n <= 96 ? 96 : n <= 128 ? 128 : 256; }

}  // namespace

namespace amica {

int plain_tile_samples() { return kS; }

int plain_pad_channels(int n) {
    return n <= 32 ? 32 : (n <= 64 ? 64 : (n <= 128 ? 128 : (n <= 256 ? 256 : -1)));
}
// Partial-sum slots per cluster: one per channel block.
int plain_partial_groups(int n) { return plain_pad_channels(n) == 256 ? PlainShape<256, 256, 1>::Q : 1; }

#define AMICA_PLAIN_EACH_M(NPV, NAV) \
    AMICA_PLAIN_CASE(NPV, NAV, 1) AMICA_PLAIN_CASE(NPV, NAV, 2) AMICA_PLAIN_CASE(NPV, NAV, 3) \
    AMICA_PLAIN_CASE(NPV, NAV, 4) AMICA_PLAIN_CASE(NPV, NAV, 5)
#define AMICA_PLAIN_EACH \
    AMICA_PLAIN_EACH_M(32, 32) AMICA_PLAIN_EACH_M(64, 64) AMICA_PLAIN_EACH_M(128, 96) \
    AMICA_PLAIN_EACH_M(128, 128) AMICA_PLAIN_EACH_M(256, 256)

int plain_max_clusters(int n, int m, int M) {
    if (plain_pad_channels(n) < 0 || m < 1 || m > 5 || M < 1 || M > kMaxModels) return -1;
    const int NA = plain_work_channels(n);
#define AMICA_PLAIN_CASE(NPV, NAV, MMV) \
    if (NA == NAV && m == MMV) return max_active_clusters<NPV, NAV, MMV>(M);
    AMICA_PLAIN_EACH
#undef AMICA_PLAIN_CASE
    return -1;
}

cudaError_t launch_estep_plain(const EStepArgs& a, int NP, int nclusters, cudaStream_t st) {
    const int NA = plain_work_channels(a.n);
#define AMICA_PLAIN_CASE(NPV, NAV, MMV) \
    if (NP == NPV && NA == NAV && a.m == MMV) return launch_plain<NPV, NAV, MMV>(a, nclusters, st);
    AMICA_PLAIN_EACH
#undef AMICA_PLAIN_CASE
    return cudaErrorInvalidValue;
}
#undef AMICA_PLAIN_EACH
#undef AMICA_PLAIN_EACH_M

// the split mixed form (128 < n <= 256) runs its density-only kernel on the
// channels this form pads to 256
bool split_form_supported(int n) { return plain_pad_channels(n) == 256; }

}  // namespace amica

namespace {

// W_hi = tf32(W) (round to nearest, ties away: the low 13 bits zero, so the
// MMA's reading of it as TF32 keeps it exactly) and W_lo = W - W_hi.
__global__ void k_split_w(const float* __restrict__ Wf, float* __restrict__ whi, float* __restrict__ wlo,
                          int64_t len) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < len; e += (int64_t)gridDim.x * blockDim.x) {
        const float w = Wf[e];
        float hi = w;
        if (isfinite(w)) hi = __uint_as_float((__float_as_uint(w) + 0x1000u) & 0xffffe000u);
        whi[e] = hi;
        wlo[e] = w - hi;
    }
}

}  // namespace

namespace amica {

cudaError_t launch_split_w(const float* Wf, float* whi, float* wlo, int64_t len, cudaStream_t st) {
    k_split_w<<<(int)std::min<int64_t>((len + 255) / 256, 1184), 256, 0, st>>>(Wf, whi, wlo, len);
    return cudaGetLastError();
}

}  // namespace amica
