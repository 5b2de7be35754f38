// FP64 device-side M-step of the AMICA EM iteration, plus the per-iteration
// preparation of the E-step constants and the deterministic reduction of the
// E-step's per-CTA partial sums.
//
// The reference runs this part as ~40 small FP64 kernels, cuBLAS/MAGMA calls
// and host round trips per iteration (src/amica.cu:835-924 and :1981-2512:
// host SVD for pinv, a synchronous bflag copy, ...).  Here it is a few small
// kernels that stay on the device, so that a whole iteration can be captured
// in one CUDA graph and no host synchronisation is needed between iterations.
#include <cooperative_groups.h>
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "common.cuh"

using namespace amica;

namespace {

namespace cg = cooperative_groups;
constexpr int kT = 256;

// ---------------------------------------------------------------------------
// k_inverse_derive: W_h = A_h^{-1}, ldet_h = -log|det A_h| and the FP32 E-step
// constants, one CTA of 512 threads per model (n <= 128).  Replaces pinv() and
// the LU log-determinant (src/amica.cu:27-127, :864-924).
//
// Gauss-Jordan elimination with partial pivoting and no row interchanges: the
// pivot of column k is a not yet used row p_k of (nearly) largest |a(p_k, k)|.
// Sweeping (p_k, k) in place,
//   a(p, k) <- 1 / a(p, k),   a(p, j) <- a(p, j) / a(p, k),
//   a(i, k) <- -a(i, k) / a(p, k),   a(i, j) <- a(i, j) - a(i, k) a(p, j) / a(p, k),
// turns column k into column p_k of P.A^{-1}, so at the end W(j, p_k) = a(p_j, k).
//
// Columns are swept in panels of 16.  Warps 0-3 sweep a panel's columns alone
// (thread r holds row r of the panel in registers): the pivot of
// column k only depends on column k as updated by the earlier pivots, and those
// updates only read the pivot rows' panel entries.  The pivot key of a row is
// the high word of |a| with its low 7 bits replaced by 127 - row (so the pivot
// is within 2^-13 of the column's largest |a|, lowest row on ties); each warp's
// best row publishes its panel row and its reciprocal (every row forms the
// reciprocal of its candidate while the warp max runs), and after one 128-thread
// barrier every thread takes the largest key, updates the next column first and
// starts the next search before the rest of its row.  What bounds the kernel is
// this chain of n dependent pivots: with one row a thread it is shorter than
// with two rows on two warps (the kernels around the E-step at n = 64: 74 -> 65
// us, n = 128: 127 -> 115, n = 32: 43 -> 39, one model).
//
// Sweeping a panel's pivots (P, K) one after another is, on the other columns
// C, the block sweep
//   a(i, C) <- [i not in P] a(i, C) + sum_t X(i, t) a_old(p_t, C),
// X being the swept panel: FP64 products on the tensor cores (mma.sync
// m8n8k4; tcgen05 has no FP64 kind) with operands in shared memory.  The
// next panel's columns get it first (all warps), then warps 4-15 apply it to
// the remaining columns while warps 0-3 sweep the next panel.
constexpr int kInvThreads = 512;
constexpr int kInvN = 128;                            // padded order
constexpr int kPanel = 16;                            // columns per panel
constexpr int kLdA = kInvN + 1;                       // odd: a warp reading a column of 32 rows hits distinct banks
constexpr int kLdX = kPanel + 4;                      // 16-byte rows; 40-word stride puts an 8 x 4 fragment on distinct banks
constexpr size_t kInvSmem = sizeof(double) * ((size_t)kInvN * kLdA + 3 * (size_t)kInvN * kLdX);

__device__ __forceinline__ void bar_panel() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// pivot key of row r holding v (0: not a candidate)
__device__ __forceinline__ uint32_t pivot_key(double v, bool usable, int r) {
    return usable ? ((((uint32_t)__double2hiint(v)) & 0x7fffff80u) | (uint32_t)(127 - r)) + 128u : 0u;
}

// a(i, 8 ct + [0, 8)) for the 16 rows tiles rt0 + [0, 8) <- [i not in P] a + X Pt^T, P the
// pivot rows of the panel at k0, X its swept columns, Pt the pivot rows' old
// entries (Pt[j][t] = a_old(p_t, j)); one warp
__device__ __forceinline__ void block_sweep_strip(double* __restrict__ As, const double* __restrict__ X,
                                                  const double* __restrict__ Pt, const int* pinv, int k0,
                                                  int ct, int rt0, int nrt, int lane) {
    const int g = lane >> 2, q = lane & 3;
    const int j = 8 * ct + 2 * q;
    double acc[8][2];
#pragma unroll
    for (int u = 0; u < 8; u++) {
        if (u < nrt) {
            const int i = 8 * (rt0 + u) + g;
            // rows pivoted in this panel have pinv in [k0, k0 + 16); other rows'
            // pinv is either not set yet or outside that range
            const bool prow = (unsigned)(pinv[i] - k0) < (unsigned)kPanel;
            acc[u][0] = prow ? 0.0 : As[i * kLdA + j];
            acc[u][1] = prow ? 0.0 : As[i * kLdA + j + 1];
        }
    }
#pragma unroll
    for (int s = 0; s < kPanel; s += 4) {
        const double bf = Pt[(8 * ct + g) * kLdX + s + q];
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (u < nrt) dmma884(acc[u][0], acc[u][1], X[(8 * (rt0 + u) + g) * kLdX + s + q], bf);
    }
#pragma unroll
    for (int u = 0; u < 8; u++) {
        if (u < nrt) {
            const int i = 8 * (rt0 + u) + g;
            As[i * kLdA + j] = acc[u][0];
            As[i * kLdA + j + 1] = acc[u][1];
        }
    }
}

__global__ void __launch_bounds__(kInvThreads, 1) k_inverse_derive(
    const double* __restrict__ A, const double* __restrict__ c, const double* __restrict__ alpha,
    const double* __restrict__ mu, const double* __restrict__ beta, const double* __restrict__ rho,
    const double* __restrict__ gm, double ldetS, double* __restrict__ W, double* __restrict__ ldet,
    double* __restrict__ ltc64, float* __restrict__ Wf, float* __restrict__ wcf,
    MixParam* __restrict__ mp, int n, int m, int NP, int* err) {
    extern __shared__ __align__(16) double smem_inv[];
    double* As = smem_inv;                            // a(r, j) at As[r * kLdA + j]
    double* Xs = As + kInvN * kLdA;                   // swept panels, two buffers: Xs[b & 1][r * kLdX + t]
    double* Pt = Xs + 2 * kInvN * kLdX;               // Pt[j * kLdX + t] = a(p_t, j) before the panel's update
    __shared__ __align__(16) double crow_v[2][4][kPanel];   // each panel warp's candidate row
    __shared__ __align__(16) uint32_t ckey[2][4];
    __shared__ double cpiv[2][4], cinv[2][4];
    __shared__ double pivs[kInvN], wcs[kInvN], cperm[kInvN], cs[kInvN];
    __shared__ float sb_cl2[kMaxMix * kInvN];      // log2 normaliser per (mixture, channel)
    __shared__ int perm[kInvN], pinv[kInvN];
    __shared__ int s_bad;
    __shared__ double s_lgm;
    const int h = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const double* Ah = A + (size_t)h * n * n;
    // columns of whole panels, and all rows that panel threads hold
    const int np16 = (n + kPanel - 1) & ~(kPanel - 1), nct = np16 / 8;
    for (int j = warp; j < np16; j += kInvThreads / 32)
#pragma unroll
        for (int u = 0; u < kInvN / 32; u++) {
            const int r = lane + 32 * u;
            As[r * kLdA + j] = (r < n && j < n) ? Ah[(size_t)j * n + r] : 0.0;
        }
    if (tid < kInvN) pinv[tid] = 0x7fffffff;
    if (tid == 0) s_bad = 0;
    // panel threads (tid < 128): row r0 = tid, not yet a pivot row
    const int r0 = tid;
    bool us0 = r0 < n;
    const int npan = (n + kPanel - 1) / kPanel;
    __syncthreads();
    for (int b = 0; b <= npan; b++) {
        const int k0 = kPanel * b;
        if (b < npan && warp < 4) {
            double* Xb = Xs + (b & 1) * kInvN * kLdX;
            double pa[kPanel];
#pragma unroll
            for (int t = 0; t < kPanel; t++) pa[t] = As[r0 * kLdA + k0 + t];
            bool bad = false;
            uint32_t key = pivot_key(pa[0], us0, r0);
            double v = pa[0];
            double rv = 1.0 / v;
            uint32_t wkey = __reduce_max_sync(0xffffffffu, key);
#pragma unroll
            for (int t = 0; t < kPanel; t++) {
                if (k0 + t >= n) break;               // uniform
                const int buf = t & 1;
                if (wkey == 0u) {
                    if (lane == 0) ckey[buf][warp] = 0u;
                } else if (key == wkey) {             // one thread: the key names its row
#pragma unroll
                    for (int j = 0; j < kPanel; j += 2)
                        *reinterpret_cast<double2*>(&crow_v[buf][warp][j]) = make_double2(pa[j], pa[j + 1]);
                    ckey[buf][warp] = key;
                    cpiv[buf][warp] = v;
                    cinv[buf][warp] = rv;
                }
                bar_panel();
                const uint4 kw = *reinterpret_cast<const uint4*>(ckey[buf]);
                const uint32_t best = max(max(kw.x, kw.y), max(kw.z, kw.w));
                const int p = 127 - (int)((best - 128u) & 127u), wb = p >> 5;
                const double piv = cpiv[buf][wb], inv = cinv[buf][wb];
                const double* pp = crow_v[buf][wb];
                const double pn = pp[t + 1 < kPanel ? t + 1 : t];
                if (best == 0u || piv == 0.0) { bad = true; break; }   // same in every panel thread
                if (tid == 0) { perm[k0 + t] = p; pinv[p] = k0 + t; pivs[k0 + t] = piv; }
                const bool is_p = r0 == p;
                us0 = us0 && !is_p;
                const double fa = pa[t] * inv;
                if (t + 1 < kPanel) {                 // the next column first, and the next search
                    pa[t + 1] = fma(-fa, pn, pa[t + 1]);
                    key = pivot_key(pa[t + 1], us0, r0);
                    v = pa[t + 1];
                    rv = 1.0 / v;
                    wkey = __reduce_max_sync(0xffffffffu, key);
                }
                double ppv[kPanel];                   // the pivot row
#pragma unroll
                for (int j = 0; j < kPanel; j += 2) {
                    const double2 d = *reinterpret_cast<const double2*>(pp + j);
                    ppv[j] = d.x;
                    ppv[j + 1] = d.y;
                }
#pragma unroll
                for (int j = 0; j < kPanel; j++)
                    if (j != t && j != t + 1) pa[j] = fma(-fa, ppv[j], pa[j]);
                pa[t] = -fa;
                if (is_p) {                           // the pivot row: its own entries over the pivot
#pragma unroll
                    for (int j = 0; j < kPanel; j++) pa[j] = j == t ? inv : ppv[j] * inv;
                }
            }
            if (bad && tid == 0) s_bad = 1;
#pragma unroll
            for (int t = 0; t < kPanel; t++) As[r0 * kLdA + k0 + t] = pa[t];
#pragma unroll
            for (int t = 0; t < kPanel; t += 2)
                *reinterpret_cast<double2*>(&Xb[r0 * kLdX + t]) = make_double2(pa[t], pa[t + 1]);
        } else if (b == 0) {
            // parameter-only work of the E-step constants, off the elimination's path
            for (int e = tid - 128; e < m * NP; e += kInvThreads - 128) {
                const int j = e / NP, i = e - j * NP;
                float cl = 0.f;
                if (i < n) {
                    const size_t idx = ((size_t)h * m + j) * n + i;
                    cl = (float)((log(alpha[idx]) + 0.5 * log(beta[idx]) - M_LN2 -
                                  lgamma(1.0 + 1.0 / rho[idx])) * 1.4426950408889634);
                }
                sb_cl2[e] = cl;
            }
            const int q = tid - 128;
            if (q < kInvN) cs[q] = q < n ? c[(size_t)h * n + q] : 0.0;
            if (q == kInvN) s_lgm = log(gm[h]);
        } else if (b >= 1 && (b == npan || warp >= 4)) {
            // the previous panel's block sweep on the columns outside it and
            // outside this panel (which got it already), in column strips of 8
            const int kp = k0 - kPanel;
            const double* Xp = Xs + ((b - 1) & 1) * kInvN * kLdX;
            const int w0 = b == npan ? 0 : 4, nw = b == npan ? 16 : 12;
            for (int ct = warp - w0; ct < nct; ct += nw) {
                const int j0 = 8 * ct;
                if ((unsigned)(j0 - kp) < (unsigned)kPanel || (unsigned)(j0 - k0) < (unsigned)kPanel) continue;
                // (constant tile counts: a runtime one doubled the kernel's time)
                int rt = 0;
                for (; rt + 8 <= nct; rt += 8) block_sweep_strip(As, Xp, Pt, pinv, kp, ct, rt, 8, lane);
                for (; rt < nct; rt += 2) block_sweep_strip(As, Xp, Pt, pinv, kp, ct, rt, 2, lane);
            }
        }
        __syncthreads();
        if (s_bad || b == npan) break;
        // Pt for this panel: its pivot rows' entries outside it, now final up to it
        const int w = min(kPanel, n - k0);
        for (int e = tid; e < kPanel * np16; e += kInvThreads) {
            const int j = e >> 4, t = e & (kPanel - 1);
            if ((unsigned)(j - k0) < (unsigned)kPanel) continue;
            Pt[j * kLdX + t] = t < w ? As[perm[k0 + t] * kLdA + j] : 0.0;
        }
        __syncthreads();
        if (b + 1 < npan) {
            // the next panel's 16 columns: 2 strips x 16 row tiles, 2 tiles per warp
            const double* Xb = Xs + (b & 1) * kInvN * kLdX;
            const int rt0 = 2 * (warp >> 1);
            if (rt0 < nct) block_sweep_strip(As, Xb, Pt, pinv, k0, 2 * (b + 1) + (warp & 1), rt0, 2, lane);
        }
        __syncthreads();
    }
    if (s_bad) {
        if (tid == 0) atomicOr(err, kErrSingular);
        return;
    }
    // W(j, q) = a(perm[j], pinv[q]).  W_h column-major: thread j = tid % 128 holds
    // its row index perm[j] and walks the columns
    double* Wh = W + (size_t)h * n * n;
    {
        const int j = tid & (kInvN - 1);
        if (j < n) {
            const double* Wr = As + perm[j] * kLdA;
#pragma unroll 4
            for (int q = tid >> 7; q < n; q += kInvThreads / kInvN) Wh[(size_t)q * n + j] = Wr[pinv[q]];
        }
    }
    if (tid < n) {
        pivs[tid] = log(fabs(pivs[tid]));
        cperm[tid] = cs[perm[tid]];                  // c at the column that holds its W column
    }
    __syncthreads();
    if (warp == 0) {
        double ld = 0.0;
        for (int k = lane; k < n; k += 32) ld += pivs[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ld += __shfl_xor_sync(0xffffffffu, ld, o);
        if (lane == 0) {
            ldet[h] = -ld;
            ltc64[h] = s_lgm - ld + ldetS;            // src/amica.cu:1009
        }
    }
    // E-step constants: W in FP32 (row-major, NP x NP, zero padded), w_c = W c,
    // and per (mixture, channel) sqrt(beta), sqrt(beta)(mu + w_c), the log2
    // normaliser and rho.  w_c(i) = sum_col a(perm[i], col) c(perm[col]): four
    // threads per row, each a quarter of the columns
    {
        const int i = tid >> 2, part = tid & 3;
        double s = 0.0;
        if (i < n) {
            const double* Wr = As + perm[i] * kLdA;
#pragma unroll 8
            for (int col = part; col < n; col += 4) s = fma(Wr[col], cperm[col], s);
        }
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        if (part == 0 && i < NP) {
            wcs[i] = s;
            wcf[(size_t)h * NP + i] = (float)s;
        }
    }
    float* Wfh = Wf + (size_t)h * NP * NP;
    {
        // NP divides the block: thread k = tid % NP keeps pinv[k] and walks the rows
        const int k = tid % NP;
        const int pk = k < n ? pinv[k] : 0;
#pragma unroll 4
        for (int i = tid / NP; i < NP; i += kInvThreads / NP)
            Wfh[(size_t)i * NP + k] = (i < n && k < n) ? (float)As[perm[i] * kLdA + pk] : 0.f;
    }
    __syncthreads();
    for (int e = tid; e < m * NP; e += kInvThreads) {
        const int j = e / NP, i = e - j * NP;
        MixParam q;
        if (i < n) {
            const size_t idx = ((size_t)h * m + j) * n + i;
            const double s = sqrt(beta[idx]);
            const double r = rho[idx];
            q.s = (float)s;
            q.off = (float)(s * (mu[idx] + wcs[i]));
            q.cl2 = sb_cl2[e];
            q.rho = (float)r;
        } else {
            q.s = 0.f; q.off = 0.f; q.cl2 = 0.f; q.rho = 1.f;
        }
        mp[((size_t)h * m + j) * NP + i] = q;
    }
}

// ---------------------------------------------------------------------------
// k_inverse_big: W_h = A_h^{-1} and log|pivots| for 128 < n <= 256, where the
// n x n FP64 matrix no longer fits in one SM's shared memory.  The blocked
// Gauss-Jordan elimination of k_inverse_derive (16-column panels, the same
// pivot keys with 8 row bits, the block sweep on the FP64 tensor cores) over a
// cluster of 8 CTAs a model, each holding the whole columns of every eighth
// panel (up to 32 columns) in shared memory.  A panel's owner sweeps it (8
// warps, one row a thread) and hands the swept panel to the others through
// global memory (32 KB, L2-resident; two buffers) and its pivot rows through
// distributed shared memory; one cluster barrier a panel.  The next panel's
// owner brings that panel up to date first, then sweeps it while everyone
// applies the block sweep to the rest.
// What bounds it is the chain of n dependent pivots and, per panel, the barrier
// and the trip through L2.  (One CTA a model on a matrix in L2, the block
// sweeps reading and writing it there, took 700 us at n = 256, M = 4; this takes
// 175, and the kernels around the E-step 294 us instead of 818.)
constexpr int kMaxN = 256;
constexpr int kBigN = kMaxN;
constexpr int kBigCtas = 8;                           // a panel each, round robin
constexpr int kBigCols = kBigN / kBigCtas;            // columns a CTA holds
constexpr int kLdS = kBigCols + 2;                    // 16-byte rows; 8 lanes reading 8 rows on distinct banks
constexpr int kLdXc = kBigN + 4;                      // column stride of X: an 8 x 4 fragment on distinct banks
constexpr size_t kBigSmem = sizeof(double) * ((size_t)kBigN * kLdS + 2 * (size_t)kPanel * kLdXc + (size_t)kBigCols * kLdX);

__device__ __forceinline__ void bar_panel8() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

__device__ __forceinline__ uint32_t pivot_key8(double v, bool usable, int r) {
    return usable ? ((((uint32_t)__double2hiint(v)) & 0x7fffff00u) | (uint32_t)(255 - r)) + 256u : 0u;
}

// block_sweep_strip for a CTA's columns: the CTA's columns 8 ct + [0, 8) of rows
// i0 + [0, 32), X column-major
__device__ __forceinline__ void block_sweep_tile(double* __restrict__ S, const double* __restrict__ X,
                                                 const double* __restrict__ Pt, const int* pinv, int k0,
                                                 int ct, int i0, int lane) {
    const int g = lane >> 2, q = lane & 3;
    double acc[4][2];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int i = i0 + 8 * u + g;
        const double2 d = *reinterpret_cast<const double2*>(&S[i * kLdS + 8 * ct + 2 * q]);
        // a row pivoted in this panel starts from zero
        const bool piv = (unsigned)(pinv[i] - k0) < (unsigned)kPanel;
        acc[u][0] = piv ? 0.0 : d.x;
        acc[u][1] = piv ? 0.0 : d.y;
    }
#pragma unroll
    for (int s = 0; s < kPanel; s += 4) {
        const double bf = Pt[(8 * ct + g) * kLdX + s + q];
#pragma unroll
        for (int u = 0; u < 4; u++) dmma884(acc[u][0], acc[u][1], X[(s + q) * kLdXc + i0 + 8 * u + g], bf);
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
        *reinterpret_cast<double2*>(&S[(i0 + 8 * u + g) * kLdS + 8 * ct + 2 * q]) = make_double2(acc[u][0], acc[u][1]);
}

__global__ void __cluster_dims__(kBigCtas, 1, 1) __launch_bounds__(kInvThreads, 1)
    k_inverse_big(const double* __restrict__ A, double* work, double* __restrict__ W,
                  double* __restrict__ pivlog, int n, int* err) {
    extern __shared__ __align__(16) double smem_big[];
    double* S = smem_big;                             // a(r, column) at S[r * kLdS + local column]
    double* Xs = S + kBigN * kLdS;                    // swept panels, two buffers: Xs[(b & 1) * 16 * kLdXc + t * kLdXc + r]
    double* Pt = Xs + 2 * kPanel * kLdXc;             // Pt[local column * kLdX + t] = a(p_t, column) before the panel's update
    __shared__ __align__(16) double crow_v[2][8][kPanel];
    __shared__ __align__(16) uint32_t ckey[2][8];
    __shared__ double cpiv[2][8], cinv[2][8];
    __shared__ double pivs[kBigCols];
    __shared__ int perm[kBigN], pinv[kBigN];
    __shared__ int s_bad[2];                          // by panel parity: a fast CTA's next panel never hides one
    cg::cluster_group cluster = cg::this_cluster();
    const int me = (int)cluster.block_rank(), h = blockIdx.x / kBigCtas;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const double* Ah = A + (size_t)h * n * n;         // column-major a(r, j) = Ah[j n + r]
    double* Xg = work + (size_t)h * 2 * kPanel * kBigN;   // two buffers, column-major
    // the global column of local column jl: panel me + 8 (jl / 16)
    auto column = [&](int jl) { return kPanel * (me + kBigCtas * (jl >> 4)) + (jl & (kPanel - 1)); };
    for (int e = tid; e < kBigCols * kBigN; e += kInvThreads) {
        const int r = e & (kBigN - 1), jl = e / kBigN, j = column(jl);
        S[r * kLdS + jl] = r < n && j < n ? Ah[(size_t)j * n + r] : 0.0;
    }
    if (tid < kBigN) pinv[tid] = 0x7fffffff;
    if (tid < 2) s_bad[tid] = 0;
    const int npan = (n + kPanel - 1) / kPanel, nrg = (n + 31) / 32;
    // the block sweep of panel `b` on the CTA's columns outside panel slot `skip`
    auto sweep_rest = [&](int b, int skip, int w0, int nw) {
        const double* Xb = Xs + (b & 1) * kPanel * kLdXc;
        for (int e = warp - w0; e < 4 * nrg; e += nw) {
            const int ct = e & 3;
            if ((ct >> 1) != skip) block_sweep_tile(S, Xb, Pt, pinv, kPanel * b, ct, 32 * (e >> 2), lane);
        }
    };
    cluster.sync();                                   // every CTA runs before the first remote store
    bool bad = false;
    for (int b = 0; b < npan; b++) {
        const int k0 = kPanel * b, slot = b / kBigCtas;
        const bool mine = b % kBigCtas == me;
        double* Xb = Xs + (b & 1) * kPanel * kLdXc;
        double* Xgb = Xg + (b & 1) * kPanel * kBigN;
        if (!mine) {
            // the previous panel's owner leaves that panel as it is
            if (b > 0) sweep_rest(b - 1, (b - 1) % kBigCtas == me ? (b - 1) / kBigCtas : -1, 0, kInvThreads / 32);
        } else if (warp >= 8) {
            if (b > 0) sweep_rest(b - 1, slot, 8, 8);   // this panel got it already
        } else {
            const int r0 = tid;                       // the thread's row, and whether no panel has pivoted it
            bool us0 = r0 < n && pinv[r0] == 0x7fffffff;
            double pa[kPanel];
#pragma unroll
            for (int t = 0; t < kPanel; t += 2) {
                const double2 d = *reinterpret_cast<const double2*>(&S[r0 * kLdS + kPanel * slot + t]);
                pa[t] = d.x;
                pa[t + 1] = d.y;
            }
            uint32_t key = pivot_key8(pa[0], us0, r0);
            double v = pa[0];
            double rv = 1.0 / v;
            uint32_t wkey = __reduce_max_sync(0xffffffffu, key);
            bool fail = false;
#pragma unroll
            for (int t = 0; t < kPanel; t++) {
                if (k0 + t >= n) break;               // uniform
                const int buf = t & 1;
                if (wkey == 0u) {
                    if (lane == 0) ckey[buf][warp] = 0u;
                } else if (key == wkey) {             // one thread: the key names its row
#pragma unroll
                    for (int j = 0; j < kPanel; j += 2)
                        *reinterpret_cast<double2*>(&crow_v[buf][warp][j]) = make_double2(pa[j], pa[j + 1]);
                    ckey[buf][warp] = key;
                    cpiv[buf][warp] = v;
                    cinv[buf][warp] = rv;
                }
                bar_panel8();
                const uint4 ka = *reinterpret_cast<const uint4*>(&ckey[buf][0]);
                const uint4 kb = *reinterpret_cast<const uint4*>(&ckey[buf][4]);
                const uint32_t best = max(max(max(ka.x, ka.y), max(ka.z, ka.w)), max(max(kb.x, kb.y), max(kb.z, kb.w)));
                const int p = 255 - (int)((best - 256u) & 255u), wb = p >> 5;
                const double piv = cpiv[buf][wb], inv = cinv[buf][wb];
                const double* pp = crow_v[buf][wb];
                const double pn = pp[t + 1 < kPanel ? t + 1 : t];
                if (best == 0u || piv == 0.0) { fail = true; break; }   // same in every panel thread
                if (tid == 0) { perm[k0 + t] = p; pivs[kPanel * slot + t] = piv; }
                const bool is_p = r0 == p;
                us0 = us0 && !is_p;
                const double fa = pa[t] * inv;
                if (t + 1 < kPanel) {                 // the next column first, and the next search
                    pa[t + 1] = fma(-fa, pn, pa[t + 1]);
                    key = pivot_key8(pa[t + 1], us0, r0);
                    v = pa[t + 1];
                    rv = 1.0 / v;
                    wkey = __reduce_max_sync(0xffffffffu, key);
                }
                double ppv[kPanel];                   // the pivot row
#pragma unroll
                for (int j = 0; j < kPanel; j += 2) {
                    const double2 d = *reinterpret_cast<const double2*>(pp + j);
                    ppv[j] = d.x;
                    ppv[j + 1] = d.y;
                }
#pragma unroll
                for (int j = 0; j < kPanel; j++)
                    if (j != t && j != t + 1) pa[j] = fma(-fa, ppv[j], pa[j]);
                pa[t] = -fa;
                if (is_p) {                           // the pivot row: its own entries over the pivot
#pragma unroll
                    for (int j = 0; j < kPanel; j++) pa[j] = j == t ? inv : ppv[j] * inv;
                }
            }
#pragma unroll
            for (int t = 0; t < kPanel; t++) {
                Xgb[t * kBigN + r0] = pa[t];
                Xb[t * kLdXc + r0] = pa[t];
            }
#pragma unroll
            for (int t = 0; t < kPanel; t += 2)
                *reinterpret_cast<double2*>(&S[r0 * kLdS + kPanel * slot + t]) = make_double2(pa[t], pa[t + 1]);
            bar_panel8();                             // perm is written
            const int q = tid / kPanel, t = tid % kPanel;   // to CTA q: pivot row t
            if (q < kBigCtas) {
                if (fail && t == 0) cluster.map_shared_rank(s_bad, q)[b & 1] = 1;
                if (!fail && q != me && k0 + t < n) cluster.map_shared_rank(perm, q)[k0 + t] = perm[k0 + t];
            }
        }
        cluster.sync();
        if (s_bad[b & 1]) { bad = true; break; }      // the same in every CTA
        if (!mine) {
            for (int e = tid; e < kPanel * kBigN / 2; e += kInvThreads) {
                double2 d;                            // from L2, and not before the barrier
                asm volatile("ld.global.cg.v2.f64 {%0, %1}, [%2];"
                             : "=d"(d.x), "=d"(d.y) : "l"(Xgb + 2 * e) : "memory");
                const int t = e / (kBigN / 2), r = 2 * (e % (kBigN / 2));
                *reinterpret_cast<double2*>(&Xb[t * kLdXc + r]) = d;
            }
        }
        // Pt for this panel: its pivot rows' entries in this CTA, final up to it
        static_assert(kPanel * kBigCols == kInvThreads, "one entry of Pt a thread");
        {
            const int jl = tid / kPanel, t = tid % kPanel;
            Pt[jl * kLdX + t] = k0 + t < n ? S[perm[k0 + t] * kLdS + jl] : 0.0;
        }
        if (tid < kPanel && k0 + tid < n) pinv[perm[k0 + tid]] = k0 + tid;
        __syncthreads();
        if (b + 1 < npan && (b + 1) % kBigCtas == me) {
            // the next panel's columns first
            const int s1 = (b + 1) / kBigCtas;
            if ((warp >> 1) < nrg) block_sweep_tile(S, Xb, Pt, pinv, k0, 2 * s1 + (warp & 1), 32 * (warp >> 1), lane);
            __syncthreads();
        }
    }
    if (bad) {
        if (me == 0 && tid == 0) atomicOr(err, kErrSingular);
        return;
    }
    sweep_rest(npan - 1, (npan - 1) % kBigCtas == me ? (npan - 1) / kBigCtas : -1, 0, kInvThreads / 32);
    __syncthreads();
    // W(j, q) = a(perm[j], pinv[q]), column-major W_h: column perm[k] from column k
    double* Wh = W + (size_t)h * n * n;
    const int j = tid & (kBigN - 1);
    if (j < n) {
        const double* Sr = S + perm[j] * kLdS;
        for (int jl = tid / kBigN; jl < kBigCols; jl += kInvThreads / kBigN) {
            const int k = column(jl);
            if (k < n) Wh[(size_t)perm[k] * n + j] = Sr[jl];
        }
    }
    if (tid < kBigCols && column(tid) < n) pivlog[(size_t)h * n + column(tid)] = log(fabs(pivs[tid]));
}

// k_derive: log|det W_h|, the Lt constant and the FP32 E-step constants from a
// column-major W (the tail of k_inverse_derive for the n > 128 path).  A CTA of 8
// warps owns 32 channels of one model: w_c = W c (warps share the columns), its
// rows of W in FP32 (32 x 32 tiles turned in shared memory) and its channels'
// mixture constants.  (One CTA per model, walking rows of the column-major W and
// adding the pivots' logarithms in one thread, took 166 us at n = 256.)
__global__ void __launch_bounds__(256) k_derive(
    const double* __restrict__ W, const double* __restrict__ pivlog, const double* __restrict__ c,
    const double* __restrict__ alpha, const double* __restrict__ mu, const double* __restrict__ beta,
    const double* __restrict__ rho, const double* __restrict__ gm, double ldetS,
    double* __restrict__ ldet, double* __restrict__ ltc64, float* __restrict__ Wf,
    float* __restrict__ wcf, MixParam* __restrict__ mp, int n, int m, int NP) {
    __shared__ double part[8][32];
    __shared__ float tile[32][33];
    const int h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int i0 = 32 * blockIdx.x, i = i0 + lane;
    const double* Wh = W + (size_t)h * n * n;
    if (blockIdx.x == 0 && warp == 0) {
        double ld = 0.0;
        for (int k = lane; k < n; k += 32) ld += pivlog[(size_t)h * n + k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ld += __shfl_xor_sync(0xffffffffu, ld, o);
        if (lane == 0) {
            ldet[h] = -ld;
            ltc64[h] = log(gm[h]) - ld + ldetS;        // src/amica.cu:1009
        }
    }
    double wc = 0.0;
    if (i < n) {
#pragma unroll 8
        for (int k = warp; k < n; k += 8) wc = fma(Wh[(size_t)k * n + i], c[(size_t)h * n + k], wc);
    }
    part[warp][lane] = wc;
    float* Wfh = Wf + (size_t)h * NP * NP;
    for (int k0 = 0; k0 < NP; k0 += 32) {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int k = k0 + warp + 8 * q;           // column k of W, rows i0 ..
            tile[lane][warp + 8 * q] = (i < n && k < n) ? (float)Wh[(size_t)k * n + i] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; q++) Wfh[(size_t)(i0 + warp + 8 * q) * NP + k0 + lane] = tile[warp + 8 * q][lane];
    }
    wc = 0.0;
#pragma unroll
    for (int w = 0; w < 8; w++) wc += part[w][lane];   // in every warp
    if (warp == 0) wcf[(size_t)h * NP + i] = (float)wc;
    if (warp < m) {
        MixParam q;
        if (i < n) {
            const size_t idx = ((size_t)h * m + warp) * n + i;
            const double s = sqrt(beta[idx]);
            const double r = rho[idx];
            q.s = (float)s;
            q.off = (float)(s * (mu[idx] + wc));
            q.cl2 = (float)((log(alpha[idx]) + 0.5 * log(beta[idx]) - M_LN2 - lgamma(1.0 + 1.0 / r)) *
                            1.4426950408889634);
            q.rho = (float)r;
        } else {
            q.s = 0.f; q.off = 0.f; q.cl2 = 0.f; q.rho = 1.f;
        }
        mp[((size_t)h * m + warp) * NP + i] = q;
    }
}

// Entry (r, cc) of the A-update matrix B_h (src/amica.cu:2155-2279,
// src/kernels.cu:961-1014): the Newton form when this model takes the Newton
// step, else the natural gradient I - phi / vsum.
__device__ __forceinline__ double b_entry(const double* __restrict__ phi, double ivs,
                                          const double* __restrict__ kappa,
                                          const double* __restrict__ lambda,
                                          const double* __restrict__ sig2, int newton, int r, int cc,
                                          int n) {
    const double prc = phi[(size_t)cc * n + r] * ivs;      // phi(r, c) / vsum
    if (newton) {
        if (r == cc) return (1.0 - prc) / lambda[r];
        const double pcr = phi[(size_t)r * n + cc] * ivs;
        const double nom = -sig2[r] * kappa[cc];
        return (nom * (-prc) + (-pcr)) / ((kappa[r] * sig2[r]) * (kappa[cc] * sig2[cc]) - 1.0);
    }
    return (r == cc ? 1.0 : 0.0) - prc;
}

// Batched FP64 32x32-tiled products on n x n column-major matrices, one
// (tile, model) per CTA of 256 threads:
//   kind 0 (A update, src/amica.cu:2330-2342):  Out = X + s_h X B_h,
//          s_h = +lrate (Newton) or -lrate (natural gradient), B_h formed
//          on the fly from phi, kappa, lambda and sigma2
//   kind 1 (phi from Psi):  Out = (Psi - gsum c^T) W^T, written into the
//          statistics vector's phi block
//   kind 2 (adjoint):  Out = vsum A^T - phi A^T, phi and vsum from the sums of
//          the gradient sweep (dL/dW_h; src/amica.cu:1535-1550 forms phi only)
struct GemmArgs {
    int kind, n, m;
    const double* X; size_t strideX;
    const double* Y; size_t strideY;        // kind 1: W, kind 2: A
    double* Out; size_t strideOut;
    const double* gs; size_t strideG;       // kind 1
    const double* c;                        // kind 1
    const int* use_newton;                  // kind 0
    const Ctrl* ctrl;                       // kind 0
    const double* stats;                    // kind 0: phi and vsum
    const double* work;                     // kind 0: kappa, lambda, sigma2
    const double* vsum; size_t strideV;     // kind 2
};

__global__ void __launch_bounds__(256) k_gemm64(GemmArgs g) {
    __shared__ double xs[32][33], ys[32][33];
    const int n = g.n;
    const int h = blockIdx.z;
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;   // ty: 0..7
    const double* Xh = g.X + g.strideX * h;
    const double* Yh = g.kind != 0 ? g.Y + g.strideY * h : nullptr;
    StatLayout SL{n, g.m};
    const double* phi = g.kind == 0 ? g.stats + SL.base(h) + SL.phi() : nullptr;
    const double ivs = g.kind == 0 ? 1.0 / g.stats[SL.base(h) + SL.vs()] : 0.0;
    const double* kappa = g.kind == 0 ? g.work + (size_t)h * 4 * n : nullptr;
    const int newton = g.kind == 0 ? g.use_newton[h] : 0;
    if (newton < 0) {                                 // frozen model: A unchanged
        const int r = r0 + tx;
        for (int q = 0; q < 4; q++) {
            const int col = c0 + ty + 8 * q;
            if (r < n && col < n) g.Out[g.strideOut * h + (size_t)col * n + r] = Xh[(size_t)col * n + r];
        }
        return;
    }
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int k0 = 0; k0 < n; k0 += 32) {
        for (int q = 0; q < 4; q++) {
            const int rr = ty + 8 * q;                 // tile-local k (for X) / k (for Y)
            // X(r0 + tx, k0 + rr)
            const int r = r0 + tx, k = k0 + rr;
            double xv = 0.0;
            if (r < n && k < n) {
                xv = Xh[(size_t)k * n + r];
                if (g.kind == 1) xv -= g.gs[g.strideG * h + r] * g.c[(size_t)h * n + k];
            }
            xs[tx][rr] = xv;
            // Y(k0 + rr, c0 + tx): kind 0 -> B_h(k, col); kinds 1, 2 -> Y^T(k, col) = Y(col, k)
            const int col = c0 + tx;
            double yv = 0.0;
            if (k < n && col < n)
                yv = (g.kind == 0) ? b_entry(phi, ivs, kappa, kappa + n, kappa + 2 * n, newton, k, col, n)
                                   : Yh[(size_t)k * n + col];
            ys[rr][tx] = yv;
        }
        __syncthreads();
#pragma unroll 8
        for (int kk = 0; kk < 32; kk++) {
            const double xv = xs[tx][kk];
#pragma unroll
            for (int q = 0; q < 4; q++) acc[q] += xv * ys[kk][ty + 8 * q];
        }
        __syncthreads();
    }
    const int r = r0 + tx;
    if (r >= n) return;
    double s = 1.0;
    if (g.kind == 0) s = newton ? g.ctrl->lrate : -g.ctrl->lrate;
    for (int q = 0; q < 4; q++) {
        const int col = c0 + ty + 8 * q;
        if (col >= n) continue;
        double* o = g.Out + g.strideOut * h + (size_t)col * n + r;
        if (g.kind == 0) *o = Xh[(size_t)col * n + r] + s * acc[q];
        else if (g.kind == 1) *o = acc[q];
        else *o = g.vsum[g.strideV * h] * Yh[(size_t)r * n + col] - acc[q];
    }
}

// Reparametrisation and c update after the A update (src/amica.cu:2367-2512):
// unit columns of A, mu *= norm, beta /= norm^2, mu -= W_old (cnew - c), c = cnew;
// and the finiteness check of everything the M-step wrote (the host then rolls
// the iteration back; the next E-step would otherwise carry NaN into the LL).
//
// A CTA of 8 warps owns 8 channels of one model: a warp its column of A (norm,
// scaled copy) and that channel's mu and beta; the CTA's rows of W (cnew - c) are
// summed by all its threads, 64 contiguous bytes of W per column.  The last CTA
// of the grid writes c (which the others read).  Bound by the latency of two
// passes over a column; with one CTA per model it took 36 us at n = 128 and 72 at
// n = 256 (and the check was a launch of its own).
// With phi_split = 2, ||A_new - A||_F / ||A||_F of each model (frozen models report
// nothing) is summed from the columns in order by the last CTA, which switches
// the split correction of phi on for good once a Newton iteration changed no
// model's A by more than phi_split_rel.
constexpr int kRepCh = 8;
struct ReparmArgs {
    int update_A, do_reparm, n, m, M, phi_split;
    double phi_split_rel;
    double *A, *c, *mu, *beta, *work;
    const double *Anew, *W, *alpha, *rho, *gm;
    const int* use_newton;
    Ctrl* ctrl;
    int* err;
};
__global__ void __launch_bounds__(32 * kRepCh) k_reparm(ReparmArgs a) {
    const int n = a.n, m = a.m, h = blockIdx.y;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int i0 = kRepCh * blockIdx.x, i = i0 + warp;
    double* work = a.work + (size_t)h * 4 * n;         // kappa, lambda (read by the A update before): per-column sums
    const double* cnew = work + 3 * n;
    const double* ch = a.c + (size_t)h * n;
    const bool frozen = a.use_newton[h] < 0;           // A, c, mu, beta unchanged
    bool bad = false;
    __shared__ double shift_s[8][kRepCh];
    __shared__ int last_s;
    const bool full = a.update_A && !frozen && a.do_reparm;
    if (full) {
        // shift(i) = sum_k W(i, k) (cnew - c)(k): thread (k % 32, channel)
        const int ic = tid & (kRepCh - 1);
        double s = 0.0;
        if (i0 + ic < n) {
            const double* Wi = a.W + (size_t)h * n * n + i0 + ic;
#pragma unroll 4
            for (int k = tid >> 3; k < n; k += 32) s = fma(Wi[(size_t)k * n], cnew[k] - ch[k], s);
        }
        s += __shfl_xor_sync(0xffffffffu, s, 8);
        s += __shfl_xor_sync(0xffffffffu, s, 16);
        if (lane < kRepCh) shift_s[warp][lane] = s;
    }
    __syncthreads();
    if (i < n) {
        double* Ai = a.A + (size_t)h * n * n + (size_t)i * n;
        double nrm = 1.0;
        if (a.update_A && !frozen) {
            const double* Ani = a.Anew + (size_t)h * n * n + (size_t)i * n;
            double s = 0.0, dd = 0.0, aa = 0.0;
            double v[8];                               // n <= 256: the column in registers
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int r = lane + 32 * u;
                v[u] = 0.0;
                if (r < n) {
                    v[u] = Ani[r];
                    const double o = Ai[r], d = v[u] - o;
                    s = fma(v[u], v[u], s);
                    dd = fma(d, d, dd);
                    aa = fma(o, o, aa);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                s += __shfl_xor_sync(0xffffffffu, s, o);
                dd += __shfl_xor_sync(0xffffffffu, dd, o);
                aa += __shfl_xor_sync(0xffffffffu, aa, o);
            }
            if (a.do_reparm) nrm = sqrt(s);
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int r = lane + 32 * u;
                if (r < n) {
                    const double w = a.do_reparm ? v[u] / nrm : v[u];
                    Ai[r] = w;
                    bad |= !isfinite(w);
                }
            }
            if (lane == 0) { work[i] = dd; work[n + i] = aa; }
        } else {
            for (int r = lane; r < n; r += 32) bad |= !isfinite(Ai[r]);
        }
        if (lane < m) {
            const size_t idx = ((size_t)h * m + lane) * n + i;
            double mv = a.mu[idx], bv = a.beta[idx];
            if (full) {
                double shift = 0.0;
#pragma unroll
                for (int w = 0; w < 8; w++) shift += shift_s[w][warp];
                mv = mv * nrm - shift;
                bv /= nrm * nrm;
                a.mu[idx] = mv;
                a.beta[idx] = bv;
            }
            bad |= !isfinite(mv) || !isfinite(bv) || !isfinite(a.alpha[idx]) || !isfinite(a.rho[idx]);
        }
        if (lane == 0) bad |= !isfinite(frozen ? ch[i] : cnew[i]);
    }
    if (blockIdx.x == 0 && tid == 0) bad |= !isfinite(a.gm[h]);
    if (__syncthreads_or(bad) && tid == 0) atomicOr(a.err, kErrNonFinite);
    // ---- the last CTA: c, and the relative change of A
    if (tid == 0) {
        __threadfence();
        last_s = atomicAdd((unsigned long long*)&a.ctrl->reparm_done, 1ull) ==
                 (unsigned long long)gridDim.x * gridDim.y - 1;
    }
    __syncthreads();
    if (!last_s) return;
    __threadfence();
    double mx = 0.0;
    for (int q = 0; q < a.M; q++) {
        if (a.use_newton[q] < 0) continue;
        const double* wq = a.work + (size_t)q * 4 * n;
        for (int r = tid; r < n; r += blockDim.x) a.c[(size_t)q * n + r] = wq[3 * n + r];   // src/amica.cu:2456-2462
        if (a.phi_split == 2 && a.update_A && warp == 0) {
            double dd = 0.0, aa = 0.0;
            for (int r = lane; r < n; r += 32) { dd += __ldcg(wq + r); aa += __ldcg(wq + n + r); }
            for (int o = 16; o > 0; o >>= 1) {
                dd += __shfl_xor_sync(0xffffffffu, dd, o);
                aa += __shfl_xor_sync(0xffffffffu, aa, o);
            }
            if (aa > 0.0) mx = fmax(mx, sqrt(dd / aa));
        }
    }
    if (tid == 0 && a.phi_split == 2 && a.update_A && a.ctrl->newton && mx < a.phi_split_rel) a.ctrl->phi_split = 1;
}

// ---------------------------------------------------------------------------
// k_reduce: raw[h][e] = sum over slots of partial[q][h][e], fixed order.  The
// n x n block is carried only by every psi_step-th slot (the tensor-core E-step
// keeps phi in one slot per cluster); when it already is phi it also goes
// straight into the statistics vector (oracle layout), as do the entries that a
// factor finishes: kappa * beta (src/kernels.cu:616), mu_denom * sqrt(beta) (:745)
// and rho * beta_denom (:748-750).  cnew is a product with A (finish_cn).  Replaces
// the block/device reductions of src/amica.cu:1618-1920.
//
// A CTA owns 32 consecutive entries; warp w adds slots w, w + nwarps, ... (one
// 256-byte row of each) and the warps' sums are added in order.  Bound by the
// latency of the dependent slot loop, not by the (L2-resident) partials: with
// one thread per entry the 1776 slots of a 32-channel fit took 259 us, and the
// 888 of a 64-channel one 133 us.
constexpr int kReduceMaxWarps = 32;
struct ReduceStats {             // stats null: raw sums only
    double* stats;
    const double *beta, *rho, *ltc64;
    const Ctrl* ctrl;
};
__global__ void __launch_bounds__(32 * kReduceMaxWarps) k_reduce(
    const double* __restrict__ partial, double* __restrict__ raw, ReduceStats rs, int nslots,
    int M, int n, int m, int psi_step, int psi_is_phi) {
    __shared__ double sh[kReduceMaxWarps][32];
    PartLayout PL{n, m};
    StatLayout SL{n, m};
    const int stride = PL.stride(), psi0 = PL.psi();
    const int64_t total = (int64_t)M * stride;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int64_t e = (int64_t)blockIdx.x * 32 + lane;
    const int h = (int)(e / stride);
    const int off = (int)(e - (int64_t)h * stride);
    const bool in_psi = off >= psi0;
    double s = 0.0;
    if (e < total) {
        const int step = in_psi ? psi_step : 1;
        const double* p = partial + e;
#pragma unroll 8
        for (int q = warp * step; q < nslots; q += nw * step) s += p[(size_t)q * total];
    }
    sh[warp][lane] = s;
    __syncthreads();
    if (warp != 0 || e >= total) return;
    for (int w = 1; w < nw; w++) s += sh[w][lane];
    raw[e] = s;
    if (!rs.stats) return;
    double* S = rs.stats + SL.base(h);
    if (in_psi) {
        if (psi_is_phi) S[SL.phi() + (off - psi0)] = s;
    } else if (off >= PL.mix(0)) {
        const int k = (off - PL.mix(0)) / (m * n), q = off - PL.mix(k);
        const size_t idx = (size_t)h * m * n + q;
        if (k == kKn) s *= rs.beta[idx];
        else if (k == kMd) s *= sqrt(rs.beta[idx]);
        else if (k == kBd) s *= rs.rho[idx] > 2.0 ? rs.rho[idx] : 1.0;
        S[SL.mix(k) + q] = s;
    } else if (off >= PL.s2() && off < PL.gs()) {
        S[SL.s2() + (off - PL.s2())] = s;
    } else if (off == 1) {
        S[SL.vs()] = s;
    } else if (off == 0 && h == 0) {
        rs.stats[0] = s + (double)rs.ctrl->nkeep * rs.ltc64[0];
    }
}

// cnew's numerator sum_t v x_i = (A sum_t v b)_i + vsum c_i (x - c = A b) for channel
// i = i0 + (thread % 32) of model h: the CTA's warps (of 256 or 1024 threads) share
// the columns of A; the result in warp 0.  sh: 32 x 32 doubles.
__device__ __forceinline__ double finish_cn(const double* __restrict__ R, const double* __restrict__ Ah,
                                            const double* __restrict__ c, int h, int n, int m, int i0,
                                            double (*sh)[32]) {
    PartLayout PL{n, m};
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int i = i0 + lane;
    double s = 0.0;
    if (i < n) {
#pragma unroll 4
        for (int k = warp; k < n; k += nw) s = fma(Ah[(size_t)k * n + i], R[PL.cn() + k], s);
    }
    __syncthreads();
    sh[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && i < n) {
        s = R[1] * c[(size_t)h * n + i];
        for (int w = 0; w < nw; w++) s += sh[w][lane];
    }
    return s;
}
// the statistics' cnew entries; blockIdx = (32-channel block, model)
__global__ void __launch_bounds__(kT) k_cn(const double* __restrict__ raw, const double* __restrict__ A,
                                           const double* __restrict__ c, double* __restrict__ stats, int n, int m) {
    __shared__ double sh[kT / 32][32];
    const int h = blockIdx.y, i = 32 * blockIdx.x + threadIdx.x;
    PartLayout PL{n, m};
    StatLayout SL{n, m};
    const double s = finish_cn(raw + (size_t)h * PL.stride(), A + (size_t)h * n * n, c, h, n, m, 32 * blockIdx.x, sh);
    if (threadIdx.x < 32 && i < n) stats[SL.base(h) + SL.cn() + i] = s;
}

// ---------------------------------------------------------------------------
struct MCfg {
    int n, m, M;
    int do_newton, update_rho, rho_start_iter, newt_start_iter, maxdec;
    int update_gm, update_alpha, update_A, update_mu, update_beta, do_reparm;
    int do_reject, rejstart, rejint, maxrej;
    int phi_split;
    double lratemax, lnatrate, lratefact, rholrate, rhomin, rhomax, rejsig;
};

__device__ double psi_series(double x) {
    // digamma: psi(x) = psi(x+6) - sum_{k<6} 1/(x+k), asymptotic series at x+6
    // with the Bernoulli coefficients B_2k/(2k) up to x^-18 (the method of the
    // reference's psi(), src/kernels.cu:906-929)
    const double coef[9] = {1.0 / 12.0, -1.0 / 120.0, 1.0 / 252.0, -1.0 / 240.0, 1.0 / 132.0,
                            -691.0 / 32760.0, 1.0 / 12.0, -3617.0 / 8160.0, 43867.0 / 14364.0};
    const double s = x + 6.0;
    double r = log(s) - 1.0 / (2.0 * s);
    const double s2 = s * s;
    double p = s2;
    for (int k = 0; k < 9; k++) { r -= coef[k] / p; p *= s2; }
    for (int k = 5; k >= 0; k--) r -= 1.0 / (x + k);
    return r;
}

// LL bookkeeping and the learning-rate schedule (src/amica.cu:1981-1993,
// :2281-2285).  One thread; no_newt: some model fails the Newton condition.
__device__ void update_ctrl(const MCfg& cf, const double* __restrict__ stats, Ctrl* ctrl, int no_newt,
                            IterRec* hist, int64_t hist_cap) {
    Ctrl c = *ctrl;
    const int64_t iter = c.iter + 1;
    const double ll = stats[0] / ((double)cf.n * (double)c.nkeep);
    const double lrate_print = c.lrate;
    c.ll_decreased = 0;
    if (iter > 1 && ll < c.ll_prev) {
        c.lrate *= cf.lratefact;
        c.numdec += 1;
        c.ll_decreased = 1;
        if (c.numdec > cf.maxdec) {
            c.lratemax *= cf.lratefact;
            c.numdec = 0;
        }
    }
    c.ll = ll;
    c.ll_prev = ll;
    c.newton = 0;
    if (cf.update_A) {
        const double step = c.lrate < 0.1 ? c.lrate : 0.1;
        if (iter >= cf.newt_start_iter && cf.do_newton && !no_newt) {
            c.lrate = fmin(cf.lratemax, c.lrate + step);
            c.newton = 1;
        } else {
            c.lrate = fmin(cf.lnatrate, c.lrate + step);
        }
        c.no_newt = no_newt;
    }
    c.iter = iter;
    c.last_rejected = 0;
    c.mstep_done = 0;
    c.reparm_done = 0;
    if (cf.phi_split != 2) c.phi_split = cf.phi_split;
    *ctrl = c;
    if (hist && iter - 1 < hist_cap) {
        IterRec r;
        r.ll = ll;
        r.lrate = lrate_print;
        r.iter = iter;
        r.newton = c.newton;
        r.ll_decreased = c.ll_decreased;
        r.nkeep = c.nkeep;
        r.nrejected = 0;
        r.phi_split = c.phi_split;          // the form this iteration's E-step ran
        hist[iter - 1] = r;
    }
}

// Parameter updates (src/amica.cu:1995-2154), the Newton condition
// (src/amica.cu:2155-2230) and the control block.  A CTA owns 32 channels of one
// model: lane = channel, warp = mixture; kappa, lambda, sigma2 and cnew go to
// `work` for the A update.  Everything is per channel but the Newton condition:
// (kappa sigma2)(kappa sigma2)^T has an entry <= 1 iff some kappa sigma2 (they are
// not negative) is <= 1 itself, the diagonal being part of it.  The last CTA of
// the grid combines the channels' findings and advances the control block.
// Bound by the latency of one chain of loads, divisions and a digamma; with one
// CTA per model walking all channels and the n^2 products, and the control block
// in a launch of its own, the two took 16 us at n = 32 and 17 at n = 128.
// raw not null: cnew's numerator comes from the E-step's raw sums (finish_cn), the
// statistics' own entries for it are not read.
constexpr int kMT = 256;
__global__ void __launch_bounds__(kMT) k_mstep(
    MCfg cf, const double* __restrict__ stats, const double* __restrict__ raw, const double* __restrict__ A,
    const double* __restrict__ c, Ctrl* ctrl, double* gm, double* alpha, double* mu, double* beta, double* rho,
    double* work, int64_t* bflag, int* use_newton, IterRec* hist, int64_t hist_cap) {
    __shared__ double sh[kMT / 32][32], kap_s[5][32], lam_s[5][32];
    __shared__ int last_s;
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, j = tid >> 5;
    const int n = cf.n, m = cf.m, mn = m * n;
    const int i = 32 * blockIdx.x + lane;
    StatLayout SL{n, m};
    PartLayout PL{n, m};
    const double* S = stats + SL.base(h);
    const int64_t iter = ctrl->iter + 1;
    const double Tk = (double)ctrl->nkeep;
    const double vsum = S[SL.vs()];
    const double ivs = 1.0 / vsum;
    const bool frozen = !(vsum >= kMinModelVsum);      // a model that explains no data
    if (blockIdx.x == 0 && tid == 0 && cf.update_gm) gm[h] = frozen ? fmax(vsum / Tk, kMinGm) : vsum / Tk;
    if (!frozen) {
        double* kappa = work + (size_t)h * 4 * n;
        double cn = 0.0;
        if (raw) cn = finish_cn(raw + (size_t)h * PL.stride(), A + (size_t)h * n * n, c, h, n, m, 32 * blockIdx.x, sh);
        if (j < m) {
            double kap = 0.0, lam = 0.0;
            if (i < n) {
                const int mi = j * n + i;
                const size_t idx = (size_t)h * mn + mi;
                const double us = S[SL.mix(kUs) + mi], kn = S[SL.mix(kKn) + mi], ln = S[SL.mix(kLn) + mi];
                const double muv = mu[idx], bv = beta[idx], rv = rho[idx];
                // alpha = usum / vsum; kappa / lambda with the new alpha and old mu
                const double al = cf.update_alpha ? us * ivs : alpha[idx];
                if (cf.update_alpha) alpha[idx] = al;
                if (us > 0.0) {                        // else a component with no responsibility: mu, beta, rho kept
                    const double dk = kn / us;
                    kap = dk * al;
                    lam = (muv * muv * dk + ln / us) * al;
                    if (cf.update_mu) mu[idx] = muv + S[SL.mix(kMn) + mi] / S[SL.mix(kMd) + mi];
                    if (cf.update_beta) beta[idx] = bv * ((rv > 2.0 ? 0.0 : us) / S[SL.mix(kBd) + mi]);
                    if (cf.update_rho && iter >= cf.rho_start_iter) {
                        const double ps = psi_series(1.0 + 1.0 / rv);
                        const double d = 1.0 - (rv / ps) * S[SL.mix(kRn) + mi] / us;
                        double r = rv + cf.rholrate * d;
                        if (r > cf.rhomax) r = cf.rhomax;
                        else if (r < cf.rhomin) r = cf.rhomin;
                        rho[idx] = r;
                    }
                }
            }
            kap_s[j][lane] = kap;
            lam_s[j][lane] = lam;
        }
        __syncthreads();
        if (j == 0) {
            bool low = false;
            if (i < n) {
                const double s2 = S[SL.s2() + i] * ivs;
                if (!raw) cn = S[SL.cn() + i];
                double kap = 0.0, lam = 0.0;
                for (int q = 0; q < m; q++) { kap += kap_s[q][lane]; lam += lam_s[q][lane]; }
                kappa[i] = kap;
                kappa[n + i] = lam;
                kappa[2 * n + i] = s2;
                kappa[3 * n + i] = cn * ivs;
                low = kap * s2 <= 1.0;
            }
            if (__any_sync(0xffffffffu, low) && lane == 0)
                atomicOr((unsigned long long*)&bflag[h], 1ull);
        }
    }
    // ---- the last CTA
    __threadfence();
    __syncthreads();
    if (tid == 0)
        last_s = atomicAdd((unsigned long long*)&ctrl->mstep_done, 1ull) ==
                 (unsigned long long)gridDim.x * gridDim.y - 1;
    __syncthreads();
    if (!last_s || tid != 0) return;
    __threadfence();
    int no_newt = 0;
    for (int q = 0; q < cf.M; q++) {
        const bool fz = !(stats[SL.base(q) + SL.vs()] >= kMinModelVsum);
        const int low = (int)atomicExch((unsigned long long*)&bflag[q], 0ull);   // zero for the next iteration
        no_newt |= low;
        use_newton[q] = fz ? -1 : cf.update_A && !low && cf.do_newton && iter >= cf.newt_start_iter;
    }
    update_ctrl(cf, stats, ctrl, no_newt, hist, hist_cap);
}

// Rejection pass (engine-defined; the reference has none): over kept samples,
// mean and std (n-1) of P in FP64, 4096-sample chunks summed in order, then the
// chunk sums in order; drop kept samples with P < mean - rejsig * std.  Runs
// only on the iterations the schedule selects.
//
// Each chunk is one CTA: its samples are loaded by all threads and laid out in
// shared memory as FP64 terms, a dropped sample as -0 (x + -0 is x for every x),
// and one thread adds them in order: the order of the sum is part of the rule,
// so the chain of 4096 dependent FP64 additions is what bounds a pass.  The last
// CTA to finish (ws->done) adds the chunk sums.  Three launches: the mean, the
// second moment and threshold, the mask.  One CTA of one thread per chunk, which
// read its samples from global memory one by one, took 1517 us at T = 300,000.
constexpr int kRejChunk = 4096;
struct RejectWs {            // after the chunk sums and chunk counts in the buffer `chunk`
    double mean, thr;
    long long nkept, dropped;
    unsigned done[3];
};
__device__ __forceinline__ RejectWs* reject_ws(double* chunk, int64_t T) {
    return reinterpret_cast<RejectWs*>(chunk + 2 * ((T + kRejChunk - 1) / kRejChunk));
}
// ctrl is not written before every CTA of the mask pass has read it here
__device__ __forceinline__ bool reject_due(const MCfg& cf, const Ctrl* ctrl, int force) {
    const int64_t it = ctrl->iter;
    return force || (cf.do_reject && ctrl->rej_passes < cf.maxrej && it >= cf.rejstart &&
                     ((it - cf.rejstart) % (cf.rejint > 0 ? cf.rejint : 1)) == 0);
}
// true in every thread of the CTA that is the last of the grid to call this
__device__ __forceinline__ bool last_cta(unsigned* done) {
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (last) __threadfence();
    return last != 0;
}

// PASS 0: chunk sums of P and counts, then the mean; PASS 1: chunk sums of
// (P - mean)^2, then the threshold.
template <int PASS>
__global__ void __launch_bounds__(kT) k_reject_sum(MCfg cf, Ctrl* ctrl, const float* __restrict__ P,
                                                   const uint8_t* __restrict__ keep, int64_t T, double* chunk,
                                                   int force) {
    if (!reject_due(cf, ctrl, force)) return;
    __shared__ __align__(16) double term[kRejChunk];
    __shared__ int cnt_s;
    const int tid = threadIdx.x;
    const int64_t nch = (T + kRejChunk - 1) / kRejChunk;
    RejectWs* ws = reject_ws(chunk, T);
    long long* cnt = reinterpret_cast<long long*>(chunk + nch);
    if (PASS == 1 && *(volatile long long*)&ws->nkept < 2) return;
    const double mean = PASS == 1 ? *(volatile double*)&ws->mean : 0.0;
    const int64_t t0 = (int64_t)blockIdx.x * kRejChunk;
    const int len = (int)(T - t0 < kRejChunk ? T - t0 : kRejChunk);
    const int padded = (len + 7) & ~7;
    if (tid == 0) cnt_s = 0;
    __syncthreads();
    int k = 0;
    for (int i = tid; i < padded; i += kT) {
        double v = -0.0;
        if (i < len && keep[t0 + i]) {
            v = (double)P[t0 + i];
            if (PASS == 1) {
                const double d = __dsub_rn(v, mean);
                v = __dmul_rn(d, d);
            }
            k++;
        }
        term[i] = v;
    }
    if (PASS == 0 && k) atomicAdd(&cnt_s, k);
    __syncthreads();
    if (tid == 0) {
        double s = 0.0;
        const double2* t2 = reinterpret_cast<const double2*>(term);
#pragma unroll 4
        for (int i = 0; i < padded / 2; i++) {
            const double2 v = t2[i];
            s = __dadd_rn(__dadd_rn(s, v.x), v.y);
        }
        chunk[blockIdx.x] = s;
        if (PASS == 0) cnt[blockIdx.x] = cnt_s;
    }
    if (!last_cta(&ws->done[PASS])) return;
    // the chunk sums in order, through shared memory
    double s = 0.0;
    long long n = 0;
    for (int64_t q0 = 0; q0 < nch; q0 += kT) {
        const int w = (int)(nch - q0 < kT ? nch - q0 : kT);
        __syncthreads();
        if (tid < w) {
            term[tid] = __ldcg(chunk + q0 + tid);
            term[kT + tid] = __longlong_as_double(__ldcg(cnt + q0 + tid));
        }
        __syncthreads();
        if (tid == 0)
            for (int q = 0; q < w; q++) {
                s = __dadd_rn(s, term[q]);
                n += __double_as_longlong(term[kT + q]);
            }
    }
    if (tid != 0) return;
    if (PASS == 0) {
        ws->nkept = n;
        ws->mean = (n > 0) ? __ddiv_rn(s, (double)n) : 0.0;
    } else {
        const double sd = __dsqrt_rn(__ddiv_rn(s, (double)(n - 1)));
        ws->thr = __dsub_rn(mean, __dmul_rn(cf.rejsig, sd));
        ctrl->rej_mean = mean;
        ctrl->rej_std = sd;
    }
    ws->done[PASS] = 0;
}

__global__ void __launch_bounds__(kT) k_reject_mask(MCfg cf, Ctrl* ctrl, const float* __restrict__ P,
                                                    uint8_t* keep, int64_t T, double* chunk, IterRec* hist,
                                                    int64_t hist_cap, int force) {
    if (!reject_due(cf, ctrl, force)) return;
    RejectWs* ws = reject_ws(chunk, T);
    if (*(volatile long long*)&ws->nkept < 2) return;
    const double thr = *(volatile double*)&ws->thr;
    int dropped = 0;
    for (int64_t t = blockIdx.x * (int64_t)kT + threadIdx.x; t < T; t += (int64_t)gridDim.x * kT)
        if (keep[t] && (double)P[t] < thr) { keep[t] = 0; dropped++; }
    dropped = __reduce_add_sync(0xffffffffu, dropped);
    if ((threadIdx.x & 31) == 0 && dropped) atomicAdd((unsigned long long*)&ws->dropped, (unsigned long long)dropped);
    if (!last_cta(&ws->done[2])) return;
    if (threadIdx.x == 0) {
        const int64_t d = (int64_t)atomicAdd((unsigned long long*)&ws->dropped, 0ull);
        ctrl->nkeep -= d;
        ctrl->nrej_total += d;
        ctrl->rej_passes += 1;
        ctrl->last_rejected = d;
        const int64_t it = ctrl->iter;
        if (hist && it >= 1 && it - 1 < hist_cap) hist[it - 1].nrejected = d;
        ws->dropped = 0;
        ws->done[2] = 0;
    }
}

void reject_pass(const MCfg& cf, Ctrl* ctrl, const float* P, uint8_t* keep, int64_t T, double* chunk,
                 IterRec* hist, int64_t hist_cap, int force, cudaStream_t st) {
    const unsigned nch = (unsigned)((T + kRejChunk - 1) / kRejChunk);
    k_reject_sum<0><<<nch, kT, 0, st>>>(cf, ctrl, P, keep, T, chunk, force);
    k_reject_sum<1><<<nch, kT, 0, st>>>(cf, ctrl, P, keep, T, chunk, force);
    const unsigned grid = (unsigned)std::min<int64_t>((T + 4 * kT - 1) / (4 * kT), 592);
    k_reject_mask<<<grid, kT, 0, st>>>(cf, ctrl, P, keep, T, chunk, hist, hist_cap, force);
}

}  // namespace

namespace amica {

// doubles of the rejection pass's workspace (zeroed once): chunk sums, chunk
// counts and the counters that each pass leaves at zero
size_t reject_ws_len(int64_t T) { return 2 * ((T + kRejChunk - 1) / kRejChunk) + (sizeof(RejectWs) + 7) / 8; }

static MCfg to_mcfg(const MStepCfgHost& h) {
    MCfg c;
    c.n = h.n; c.m = h.m; c.M = h.M;
    c.do_newton = h.do_newton; c.update_rho = h.update_rho; c.rho_start_iter = h.rho_start_iter;
    c.newt_start_iter = h.newt_start_iter; c.maxdec = h.maxdec; c.update_gm = h.update_gm;
    c.update_alpha = h.update_alpha; c.update_A = h.update_A; c.update_mu = h.update_mu;
    c.update_beta = h.update_beta; c.do_reparm = h.do_reparm; c.do_reject = h.do_reject;
    c.rejstart = h.rejstart; c.rejint = h.rejint; c.maxrej = h.maxrej; c.phi_split = h.phi_split;
    c.lratemax = h.lratemax; c.lnatrate = h.lnatrate; c.lratefact = h.lratefact;
    c.rholrate = h.rholrate; c.rhomin = h.rhomin; c.rhomax = h.rhomax; c.rejsig = h.rejsig;
    return c;
}

cudaError_t launch_prep(const MStepBuffers& b, const MStepCfgHost& h, cudaStream_t st) {
    if (h.n > kMaxN) return cudaErrorInvalidValue;
    if (h.n > 128) {
        if (!b.gj) return cudaErrorInvalidValue;
        double* pivlog = b.gj + (size_t)h.M * h.n * h.n;
        cudaError_t e = cudaFuncSetAttribute(k_inverse_big, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)kBigSmem);
        if (e != cudaSuccess) return e;
        k_inverse_big<<<kBigCtas * h.M, kInvThreads, kBigSmem, st>>>(b.A, b.gj, b.W, pivlog, h.n, b.err);
        k_derive<<<dim3(h.NP / 32, h.M), 256, 0, st>>>(b.W, pivlog, b.c, b.alpha, b.mu, b.beta, b.rho, b.gm, h.ldetS,
                                      b.ldet, b.ltc64, b.Wf, b.wcf, b.mp, h.n, h.m, h.NP);
        return cudaGetLastError();
    }
    if (h.NP > 128 || kInvThreads % h.NP || h.m > kMaxMix) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(k_inverse_derive, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kInvSmem);
    if (e != cudaSuccess) return e;
    k_inverse_derive<<<h.M, kInvThreads, kInvSmem, st>>>(b.A, b.c, b.alpha, b.mu, b.beta, b.rho, b.gm,
                                                     h.ldetS, b.W, b.ldet, b.ltc64, b.Wf, b.wcf, b.mp,
                                                     h.n, h.m, h.NP, b.err);
    return cudaGetLastError();
}

// Warps per CTA: about 16 slots each, so that a warp's loop is two batches of eight
// independent loads (4 warps at the least, to fill the SMs' load queues).
static cudaError_t reduce_slots(const double* partial, double* raw, const ReduceStats& rs, int nslots, int M, int n,
                                int m, int psi_step, int psi_is_phi, cudaStream_t st) {
    PartLayout PL{n, m};
    const int64_t total = (int64_t)M * PL.stride();
    int nw = 4;
    while (nw < kReduceMaxWarps && nw * 16 < nslots) nw *= 2;
    k_reduce<<<(unsigned)((total + 31) / 32), 32 * nw, 0, st>>>(partial, raw, rs, nslots, M, n, m, psi_step,
                                                                psi_is_phi);
    return cudaGetLastError();
}

// the slot sums alone (adjoint.cu)
cudaError_t launch_reduce(const double* partial, double* raw, int nslots, int M, int n, int m, int psi_step,
                          cudaStream_t st) {
    return reduce_slots(partial, raw, ReduceStats{}, nslots, M, n, m, psi_step, 0, st);
}

// The statistics from the partial slots.  with_cn = false leaves their cnew
// entries to launch_mstep(cn_from_raw).
cudaError_t launch_reduce_finalize(const MStepBuffers& b, const MStepCfgHost& h, int nslots, bool with_cn,
                                   cudaStream_t st) {
    PartLayout PL{h.n, h.m};
    StatLayout SL{h.n, h.m};
    const ReduceStats rs{b.stats, b.beta, b.rho, b.ltc64, b.ctrl};
    cudaError_t e = reduce_slots(b.partial, b.raw, rs, nslots, h.M, h.n, h.m, h.psi_step > 0 ? h.psi_step : 1,
                                 h.psi_is_phi, st);
    if (e != cudaSuccess) return e;
    if (with_cn) k_cn<<<dim3((h.n + 31) / 32, h.M), kT, 0, st>>>(b.raw, b.A, b.c, b.stats, h.n, h.m);
    if (!h.psi_is_phi) {
        dim3 g((h.n + 31) / 32, (h.n + 31) / 32, h.M);
        GemmArgs ga{};
        ga.kind = 1; ga.n = h.n; ga.m = h.m;
        ga.X = b.raw + PL.psi(); ga.strideX = PL.stride();
        ga.Y = b.W; ga.strideY = (size_t)h.n * h.n;
        ga.Out = b.stats + SL.base(0) + SL.phi(); ga.strideOut = SL.S();
        ga.gs = b.raw + PL.gs(); ga.strideG = PL.stride();
        ga.c = b.c;
        k_gemm64<<<g, 256, 0, st>>>(ga);
    }
    return cudaGetLastError();
}

// dL/dW_h = vsum W^{-T} - phi W^{-T} (W^{-1} = A) from the gradient sweep's sums
// (tensor-core form, whose n x n block is phi), M matrices of n x n at out.
cudaError_t launch_adjoint_dw(const double* raw, const double* A, double* out, int n, int m, int M,
                              cudaStream_t st) {
    PartLayout PL{n, m};
    GemmArgs ga{};
    ga.kind = 2; ga.n = n; ga.m = m;
    ga.X = raw + PL.psi(); ga.strideX = PL.stride();
    ga.Y = A; ga.strideY = (size_t)n * n;
    ga.Out = out; ga.strideOut = (size_t)n * n;
    ga.vsum = raw + 1; ga.strideV = PL.stride();
    k_gemm64<<<dim3((n + 31) / 32, (n + 31) / 32, M), 256, 0, st>>>(ga);
    return cudaGetLastError();
}

// The M-step from b.stats; cn_from_raw: cnew's numerator from b.raw instead.
cudaError_t launch_mstep(const MStepBuffers& b, const MStepCfgHost& h, bool cn_from_raw, const float* P_rel,
                         uint8_t* keep, int64_t T, cudaStream_t st) {
    const MCfg cf = to_mcfg(h);
    k_mstep<<<dim3((h.n + 31) / 32, h.M), kMT, 0, st>>>(cf, b.stats, cn_from_raw ? b.raw : nullptr, b.A, b.c, b.ctrl,
                                                        b.gm, b.alpha, b.mu, b.beta, b.rho, b.work, b.bflag,
                                                        b.use_newton, b.hist, b.hist_cap);
    if (h.update_A) {
        dim3 g((h.n + 31) / 32, (h.n + 31) / 32, h.M);
        GemmArgs ga{};
        ga.kind = 0; ga.n = h.n; ga.m = h.m;
        ga.X = b.A; ga.strideX = (size_t)h.n * h.n;
        ga.Out = b.Anew; ga.strideOut = (size_t)h.n * h.n;
        ga.use_newton = b.use_newton; ga.ctrl = b.ctrl;
        ga.stats = b.stats; ga.work = b.work;
        k_gemm64<<<g, 256, 0, st>>>(ga);
    }
    ReparmArgs ra{h.update_A, h.do_reparm, h.n, h.m, h.M, h.phi_split, h.phi_split_rel,
                  b.A, b.c, b.mu, b.beta, b.work, b.Anew, b.W, b.alpha, b.rho, b.gm, b.use_newton, b.ctrl, b.err};
    k_reparm<<<dim3((h.n + kRepCh - 1) / kRepCh, h.M), 32 * kRepCh, 0, st>>>(ra);
    if (h.do_reject && P_rel && keep)
        reject_pass(cf, b.ctrl, P_rel, keep, T, b.chunk, b.hist, b.hist_cap, 0, st);
    return cudaGetLastError();
}

cudaError_t launch_reject_now(const MStepBuffers& b, const MStepCfgHost& h, const float* P_rel,
                              uint8_t* keep, int64_t T, cudaStream_t st) {
    const MCfg cf = to_mcfg(h);
    reject_pass(cf, b.ctrl, P_rel, keep, T, b.chunk, b.hist, b.hist_cap, 1, st);
    return cudaGetLastError();
}

}  // namespace amica
