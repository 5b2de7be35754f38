// Centring and sphering on the GPU in FP64 (replaces center() and whiten(),
// src/preprocess.cu:31-420 of the reference, which use a float-accumulated
// mean, cuBLAS Dsyrk and MAGMA dsyevd / dgesv / dgetrf).
//
//   mean      FP64 column sums, per-CTA partials reduced in fixed order
//   C         X_c^T X_c / T on the FP64 tensor cores (k_cov_mma)
//   S         do_sphere 1: 2 C^{-1/2} from the one-sided Jacobi of sphere_eig.cu
//             or, when C is not numerically positive definite, the two-sided
//             parallel-ordered Jacobi below;
//             do_sphere 2: diag(1/std) (std with T-1, src/kernels.cu:148-161);
//             do_sphere 0: I
//   ldetS     -log|det S| = -sum log of the eigen-scales
//   x         S (x - mean) in FP64 (tensor cores, k_apply_sphere), rounded once to FP32 into the padded
//             sample-major layout the E-step reads.
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "common.cuh"
#include "tc_ptx.cuh"

namespace amica {
// Zero floats past the T x ldx sphered data: up to three samples that fill the
// last row of 128 floats, then kXTailRows rows (256 channels: 3 rows for the
// contraction of the split form).
size_t x_tail_len(int ldx) { return ldx <= 128 ? 128 + (size_t)kXTailRows * 128 : 3 * (size_t)ldx; }
// sphere_eig.cu
cudaError_t launch_eig_cluster(const double* C, double* V, double* evals, int n, int* done, cudaStream_t st);
}  // namespace amica

namespace {

// Column sums of a contiguous run of samples per CTA: a group of ceil(n / 32)
// warps reads one sample (coalesced), the CTA's groups take samples in turn with
// eight in flight per thread, and the groups' sums are added in order.  Bound by
// HBM (0.10 ms for the 512 MB of n = 128, T = 1M); with one thread per channel and no more than n threads busy per CTA it
// took 561 us at n = 128, T = 1M (512 MB) and 569 us at n = 160, T = 50k.
constexpr int kSumThreads = 256;
__global__ void __launch_bounds__(kSumThreads) k_colsum(const float* __restrict__ x, int64_t T, int n, int64_t chunk,
                                                        double* __restrict__ part) {
    __shared__ double sh[kSumThreads];
    const int width = (n + 31) & ~31;                  // <= kSumThreads
    const int ngrp = kSumThreads / width;
    const int grp = threadIdx.x / width, i = threadIdx.x - grp * width;
    const int64_t t0 = (int64_t)blockIdx.x * chunk;
    const int64_t t1 = t0 + chunk < T ? t0 + chunk : T;
    double s = 0.0;
    if (grp < ngrp && i < n) {
        int64_t t = t0 + grp;
        for (; t + 7 * ngrp < t1; t += 8 * ngrp) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = x[(t + u * ngrp) * n + i];
#pragma unroll
            for (int u = 0; u < 8; u++) s += (double)v[u];
        }
        for (; t < t1; t += ngrp) s += (double)x[t * n + i];
    }
    sh[threadIdx.x] = s;
    __syncthreads();
    if (grp == 0 && i < n) {
        for (int g = 1; g < ngrp; g++) s += sh[g * width + i];
        part[(size_t)blockIdx.x * n + i] = s;
    }
}

// out[e] = (sum over nblk partials of part[b * len + e], in a fixed order) / div
// for e < len: a CTA owns 32 entries, its 16 warps share the partials
constexpr int kFoldWarps = 16;
__device__ __forceinline__ double fold_partials(const double* __restrict__ part, int nblk, size_t len, size_t e,
                                                bool in) {
    __shared__ double sh[kFoldWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double s = 0.0;
    if (in) {
#pragma unroll 8
        for (int b = warp; b < nblk; b += kFoldWarps) s += part[(size_t)b * len + e];
    }
    sh[warp][lane] = s;
    __syncthreads();
    if (warp == 0)
        for (int w = 1; w < kFoldWarps; w++) s += sh[w][lane];
    return s;                                          // warp 0
}
__global__ void __launch_bounds__(32 * kFoldWarps) k_mean(const double* __restrict__ part, int nblk, int n,
                                                          double div, double* __restrict__ mean) {
    const int i = blockIdx.x * 32 + (threadIdx.x & 31);
    const double s = fold_partials(part, nblk, n, i, i < n);
    if (threadIdx.x < 32 && i < n) mean[i] = s / div;
}

// The partial covariances hold the 32 x 32 tiles on and above the diagonal.
__global__ void __launch_bounds__(32 * kFoldWarps) k_cov_reduce(const double* __restrict__ part, int nblk, int n,
                                                                double div, double* __restrict__ C) {
    const int e = blockIdx.x * 32 + (threadIdx.x & 31);
    const int i = e % n, k = e / n;                    // element (i, k) at k * n + i
    const bool in = e < n * n && (i >> 5) <= (k >> 5);
    const double s = fold_partials(part, nblk, (size_t)n * n, e, in);
    if (threadIdx.x < 32 && in) {
        C[e] = s / div;
        C[(size_t)i * n + k] = s / div;
    }
}

// The sharded form's inputs to k_sphere: the covariance (scatter / T) and, for
// do_sphere 2, the per-channel variance (scatter diagonal / (T - 1)) of all
// shards.
__global__ void k_scale_scatter(const double* __restrict__ scatter, int n, double T,
                                double* __restrict__ C, double* __restrict__ var) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n * n; e += blockDim.x * gridDim.x) {
        C[e] = scatter[e] / T;
        if (e % (n + 1) == 0) var[e / (n + 1)] = scatter[e] / (T - 1.0);
    }
}

// S = V diag(2/sqrt(d)) V^T (do_sphere 1), diag(1/std) (2) or I (0); ldetS.
// The scales are formed once per CTA (formed in the inner loop they took the
// kernel 82 us at n = 128).
__global__ void __launch_bounds__(256) k_sphere(const double* __restrict__ V, const double* __restrict__ evals,
                                                const double* __restrict__ var, int n, int do_sphere,
                                                double* __restrict__ S, double* __restrict__ ldetS) {
    __shared__ double scale[256], part[8];
    const int tid = threadIdx.x;
    if (tid < n) scale[tid] = do_sphere == 1 ? 2.0 / sqrt(evals[tid]) : do_sphere == 2 ? 1.0 / sqrt(var[tid]) : 1.0;
    __syncthreads();
    for (int e = tid + blockIdx.x * blockDim.x; e < n * n; e += blockDim.x * gridDim.x) {
        const int i = e % n, k = e / n;
        double v = 0.0;
        if (do_sphere == 1) {
#pragma unroll 8
            for (int q = 0; q < n; q++) v += V[(size_t)q * n + i] * scale[q] * V[(size_t)q * n + k];
        } else {
            v = (i == k) ? scale[i] : 0.0;
        }
        S[e] = v;
    }
    if (blockIdx.x == 0) {
        double ld = tid < n ? log(scale[tid]) : 0.0;
        for (int o = 16; o > 0; o >>= 1) ld += __shfl_xor_sync(0xffffffffu, ld, o);
        if ((tid & 31) == 0) part[tid >> 5] = ld;
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < 8; w++) ld += part[w];
            *ldetS = -ld;
        }
    }
}

// per-channel variance about the (second) mean, divisor T-1 (do_sphere 2)
__global__ void k_var(const float* __restrict__ x, int64_t T, int n, const double* __restrict__ mean,
                      double* __restrict__ var) {
    const int i = blockIdx.x;
    __shared__ double sh[256];
    double s = 0.0;
    for (int64_t t = threadIdx.x; t < T; t += blockDim.x) s += (double)x[t * n + i] - mean[i];
    sh[threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int k = 0; k < (int)blockDim.x; k++) tot += sh[k];
        sh[0] = tot / (double)T;
    }
    __syncthreads();
    const double mu2 = sh[0];
    __syncthreads();
    double m2 = 0.0;
    for (int64_t t = threadIdx.x; t < T; t += blockDim.x) {
        const double d = fabs((double)x[t * n + i] - mean[i] - mu2);
        m2 += d * d;
    }
    sh[threadIdx.x] = m2;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int k = 0; k < (int)blockDim.x; k++) tot += sh[k];
        var[i] = tot / (double)(T - 1);
    }
}

// Round to the TF32 grid, nearest with ties away from zero (the tensor cores
// read only the top 19 bits of an FP32 operand, i.e. truncate; storing the data
// pre-rounded makes the TF32 contraction see an unbiased value).
__device__ __forceinline__ float round_tf32(float v) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
    return __uint_as_float(r);
}

// A stage of raw samples for the two kernels below: [t0, t0 + rows) up to T is
// one contiguous run of floats that starts on a 16-byte boundary (t0 a multiple
// of 16), so one bulk copy brings it; its size is rounded up to 16 bytes (the
// raw buffer has 16 spare bytes at its end).
__device__ __forceinline__ void load_run(float* dst, const float* x, int64_t t0, int64_t T, int rows, int n,
                                         uint64_t* bar) {
    const int64_t left = T - t0;
    const uint32_t bytes = ((uint32_t)(left < rows ? left : rows) * (uint32_t)n * 4u + 15u) & ~15u;
    mbar_expect_tx(bar, bytes);
    bulk_load(smem_u32(dst), x + t0 * n, bytes, bar);
}
// f(row, channel) over this thread's elements of a stage: the (row, 32-channel
// block) pairs warp, warp + nw, ... of rows x nb
template <class F>
__device__ __forceinline__ void each_element(int rows, int nb, int nw, F&& f) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int dr = nw / nb, db = nw - dr * nb;
    int r = warp / nb, blk = warp - r * nb;
    while (r < rows) {
        f(r, blk * 32 + lane);
        r += dr;
        blk += db;
        if (blk >= nb) { blk -= nb; r++; }
    }
}

// Partial covariance sum_t xc_t xc_t^T (xc = x - mean) in FP64 on the tensor
// cores (mma.sync m8n8k4), one persistent CTA per SM over a contiguous sample
// range.  The channels form 32 x 32 tiles of which only those on and above the
// diagonal are computed: warp = (tile, replica), a replica taking every
// nrep-th group of four samples.  A fragment (four samples of eight channels)
// has the same layout as either operand.  A stage arrives by one bulk copy during
// the products of the one before and is centred into one of two FP64 tiles (row
// stride 4 doubles modulo 16: fragment loads free of bank conflicts), so that a
// stage has one barrier and warps that are done with one tile convert into the
// other.  Bound by the FP64 pipe: at n = 128, T = 1M the ten tiles are 2.05e10
// flop, 0.56 ms at the 36.7 TFLOP/s that this instruction reaches; it takes 0.84
// ms (the FP64 pipe 59% busy with 32-sample stages, more with 64).  (The 8 x 8
// register blocking on the FMA pipe that it replaced computed all of C, in 128
// channels whatever n: 2.6 ms there, and 3.3e10 flop at n = 32 as well.)
struct CovPlan {
    int nb, ntl, nrep, ysplit, rows;   // channel blocks, tiles per CTA, replicas, CTAs per sample range, samples per stage
    int threads;
    size_t smem;
};
CovPlan cov_plan(int n) {
    CovPlan p;
    p.nb = (n + 31) / 32;
    const int tiles = p.nb * (p.nb + 1) / 2;
    p.ysplit = tiles <= 20 ? 1 : tiles == 21 ? 3 : 2;  // 20 warps of 96 registers fill an SM; 28 and 36 are even
    p.ntl = tiles / p.ysplit;
    p.nrep = p.ntl == 1 ? 8 : p.ntl == 3 ? 4 : p.ntl <= 10 ? 2 : 1;
    p.rows = p.nb == 1 ? 128 : p.nb <= 5 ? 64 : 32;
    p.threads = 32 * p.ntl * p.nrep;
    p.smem = sizeof(double) * 2 * (size_t)p.rows * (32 * p.nb + 4) + sizeof(float) * (size_t)p.rows * n;
    const size_t fold = sizeof(double) * (size_t)p.ntl * 1024;   // replicas are added through the FP64 tiles
    if (p.nrep > 1 && p.smem < fold) p.smem = fold;
    return p;
}
constexpr int kCovMaxThreads = 640;
__global__ void __launch_bounds__(kCovMaxThreads, 1) k_cov_mma(const float* __restrict__ x, int64_t T, int n,
                                                              int64_t chunk, const double* __restrict__ mean,
                                                              double* __restrict__ part, int nb, int ntl, int nrep,
                                                              int rows, int* err) {
    extern __shared__ __align__(16) double cv[];
    const int ld = 32 * nb + 4;
    double* xs = cv;                                   // [2][rows][ld], centred
    float* raw = reinterpret_cast<float*>(cv + 2 * (size_t)rows * ld);   // [rows][n]
    __shared__ double mean_s[256];
    __shared__ uint64_t bar;
    __shared__ int abort_s;
    volatile int* abort_flag = &abort_s;
    const int tid = threadIdx.x, nthr = blockDim.x, warp = tid >> 5, lane = tid & 31, nw = nthr >> 5;
    const int g = lane >> 2, q = lane & 3;
    const int rep = warp / ntl;
    int tile = warp - rep * ntl + blockIdx.y * ntl, kb = 0;
    while (tile > kb) { tile -= kb + 1; kb++; }        // column kb holds tiles (0 .. kb, kb)
    const int ib = tile;
    const int64_t t0 = (int64_t)blockIdx.x * chunk;
    const int64_t t1 = t0 + chunk < T ? t0 + chunk : T;
    for (int i = tid; i < 256; i += nthr) mean_s[i] = i < n ? mean[i] : 0.0;
    if (tid == 0) {
        abort_s = 0;
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (t0 < t1) load_run(raw, x, t0, t1, rows, n, &bar);
    }
    double acc[4][4][2];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[a][c][0] = acc[a][c][1] = 0.0;
    __syncthreads();                                   // mean_s, the barrier
    uint32_t stage = 0;
    for (int64_t tb = t0; tb < t1; tb += rows, stage++) {
        double* xb = xs + (size_t)(stage & 1) * rows * ld;
        mbar_wait(&bar, stage & 1, abort_flag, err);
        each_element(rows, nb, nw, [&](int r, int i) {
            xb[r * ld + i] = (tb + r < t1 && i < n) ? (double)raw[r * n + i] - mean_s[i] : 0.0;
        });
        __syncthreads();
        if (tid == 0 && tb + rows < t1) load_run(raw, x, tb + rows, t1, rows, n, &bar);
#pragma unroll 2
        for (int r0 = 4 * rep; r0 < rows; r0 += 4 * nrep) {
            const double* row = xb + (r0 + q) * ld + g;
            double fa[4], fb[4];
#pragma unroll
            for (int a = 0; a < 4; a++) {
                fa[a] = row[32 * ib + 8 * a];
                fb[a] = row[32 * kb + 8 * a];
            }
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int c = 0; c < 4; c++) dmma884(acc[a][c][0], acc[a][c][1], fa[a], fb[c]);
        }
    }
    // replicas into replica 0, in order
    double* fold = cv + (size_t)(warp - rep * ntl) * 1024 + lane;
    for (int w = 1; w < nrep; w++) {
        __syncthreads();
        if (rep == w) {
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int c = 0; c < 4; c++)
#pragma unroll
                    for (int u = 0; u < 2; u++) fold[((a * 4 + c) * 2 + u) * 32] = acc[a][c][u];
        }
        __syncthreads();
        if (rep == 0) {
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int c = 0; c < 4; c++)
#pragma unroll
                    for (int u = 0; u < 2; u++) acc[a][c][u] += fold[((a * 4 + c) * 2 + u) * 32];
        }
    }
    if (rep != 0) return;
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int i = 32 * ib + 8 * a + g, k = 32 * kb + 8 * c + 2 * q + u;
                if (i < n && k < n) part[(size_t)blockIdx.x * n * n + (size_t)k * n + i] = acc[a][c][u];
            }
}

// Parallel-ordered cyclic Jacobi eigendecomposition of the symmetric n x n
// matrix C (n <= 128), one CTA, everything in shared memory: the upper
// triangle of the working matrix packed by columns and the eigenvector matrix
// V.  A round applies n/2 disjoint rotations (p_k, q_k) of the round-robin
// schedule at once.  Since J^T A J only mixes rows {p_K, q_K} with columns
// {p_L, q_L}, each 2 x 2 block (K, L), K <= L, is transformed independently by
// the thread that owns it; V <- V J rotates column pairs.  Sweeps stop when the
// off-diagonal energy is below 1e-30 of the total.
__device__ __forceinline__ int pk_idx(int i, int j) {   // i <= j
    return (j * (j + 1)) / 2 + i;
}
__device__ __forceinline__ int pk_sym(int i, int j) { return i <= j ? pk_idx(i, j) : pk_idx(j, i); }

constexpr int kJacThreads = 1024;
__global__ void __launch_bounds__(kJacThreads, 1) k_jacobi_smem(const double* __restrict__ C,
                                                                double* __restrict__ Vout,
                                                                double* __restrict__ evals, int n,
                                                                const int* __restrict__ done) {
    if (*done) return;                                  // launch_eig_cluster has decomposed C
    extern __shared__ __align__(16) double jsm[];
    const int np = (n * (n + 1)) / 2;
    double* ap = jsm;                                   // packed upper triangle
    double* V = jsm + ((np + 1) & ~1);                  // n x n, column-major
    __shared__ double cs[64], sn[64];
    __shared__ int pp[64], qq[64];
    __shared__ unsigned short blkKL[64 * 65 / 2];   // (K << 8) | L for the 2 x 2 blocks, K <= L
    __shared__ double red[32];
    __shared__ int stop;
    const int tid = threadIdx.x;
    const int ne = n + (n & 1), half = ne / 2;
    const int nblk = half * (half + 1) / 2;
    for (int e = tid; e < n * n; e += kJacThreads) {
        const int r = e % n, c = e / n;
        if (r <= c) ap[pk_idx(r, c)] = C[e];
        V[e] = (r == c) ? 1.0 : 0.0;
    }
    if (tid < half)
        for (int K = 0; K <= tid; K++) blkKL[tid * (tid + 1) / 2 + K] = (unsigned short)((K << 8) | tid);
    __syncthreads();
    for (int sweep = 0; sweep < 40; sweep++) {
        double off = 0.0, tot = 0.0;
        for (int e = tid; e < np; e += kJacThreads) {
            // column j of the packed triangle holds rows 0..j; the last one is diagonal
            int j = (int)((sqrt(8.0 * e + 1.0) - 1.0) * 0.5);
            while (pk_idx(0, j + 1) <= e) j++;
            while (pk_idx(0, j) > e) j--;
            const double v = ap[e];
            const bool diag = (e - pk_idx(0, j)) == j;
            tot += diag ? v * v : 2.0 * v * v;
            off += diag ? 0.0 : 2.0 * v * v;
        }
        for (int o = 16; o > 0; o >>= 1) {
            off += __shfl_xor_sync(0xffffffffu, off, o);
            tot += __shfl_xor_sync(0xffffffffu, tot, o);
        }
        if ((tid & 31) == 0) red[tid >> 5] = off;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int w = 0; w < kJacThreads / 32; w++) s += red[w];
            red[0] = s;
        }
        __syncthreads();
        const double offt = red[0];
        __syncthreads();
        if ((tid & 31) == 0) red[tid >> 5] = tot;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int w = 0; w < kJacThreads / 32; w++) s += red[w];
            stop = (offt <= 1e-30 * s);
        }
        __syncthreads();
        if (stop) break;
        for (int round = 0; round < ne - 1; round++) {
            if (tid < half) {
                auto pos = [&](int j) { return j == 0 ? 0 : 1 + ((j - 1 + round) % (ne - 1)); };
                int p = pos(tid), q = pos(ne - 1 - tid);
                if (p > q) { const int t = p; p = q; q = t; }
                double c = 1.0, s = 0.0;
                if (q < n) {
                    const double apq = ap[pk_idx(p, q)];
                    if (fabs(apq) >= 1e-300) {
                        const double app = ap[pk_idx(p, p)], aqq = ap[pk_idx(q, q)];
                        const double th = (aqq - app) / (2.0 * apq);
                        const double t = (th >= 0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
                        c = 1.0 / sqrt(t * t + 1.0);
                        s = t * c;
                    }
                }
                pp[tid] = p; qq[tid] = q; cs[tid] = c; sn[tid] = s;
            }
            __syncthreads();
            // A <- J^T A J, one 2 x 2 block (K <= L) per work item
            for (int e = tid; e < nblk; e += kJacThreads) {
                const int K = blkKL[e] >> 8, L = blkKL[e] & 0xff;
                const int pK = pp[K], qK = qq[K], pL = pp[L], qL = qq[L];
                const double cK = cs[K], sK = sn[K], cL = cs[L], sL = sn[L];
                if (K == L) {
                    if (qK < n && sK != 0.0) {
                        const double app = ap[pk_idx(pK, pK)], aqq = ap[pk_idx(qK, qK)];
                        const double apq = ap[pk_idx(pK, qK)];
                        ap[pk_idx(pK, pK)] = cK * cK * app - 2.0 * cK * sK * apq + sK * sK * aqq;
                        ap[pk_idx(qK, qK)] = sK * sK * app + 2.0 * cK * sK * apq + cK * cK * aqq;
                        ap[pk_idx(pK, qK)] = 0.0;
                    }
                    continue;
                }
                if (sK == 0.0 && sL == 0.0) continue;
                const bool hq = qK < n, hqL = qL < n;
                const double b11 = ap[pk_sym(pK, pL)];
                const double b12 = hqL ? ap[pk_sym(pK, qL)] : 0.0;
                const double b21 = hq ? ap[pk_sym(qK, pL)] : 0.0;
                const double b22 = (hq && hqL) ? ap[pk_sym(qK, qL)] : 0.0;
                // B J_L (columns), then J_K^T (rows); J = [[c, s], [-s, c]]
                const double d11 = cL * b11 - sL * b12, d12 = sL * b11 + cL * b12;
                const double d21 = cL * b21 - sL * b22, d22 = sL * b21 + cL * b22;
                ap[pk_sym(pK, pL)] = cK * d11 - sK * d21;
                if (hqL) ap[pk_sym(pK, qL)] = cK * d12 - sK * d22;
                if (hq) ap[pk_sym(qK, pL)] = sK * d11 + cK * d21;
                if (hq && hqL) ap[pk_sym(qK, qL)] = sK * d12 + cK * d22;
            }
            // V <- V J: 16 threads per rotation, rows r = lane16, lane16 + 16, ...
            for (int k = tid >> 4; k < half; k += kJacThreads / 16) {
                const int p = pp[k], q = qq[k];
                const double s = sn[k];
                if (q >= n || s == 0.0) continue;
                const double c = cs[k];
                for (int r = tid & 15; r < n; r += 16) {
                    const double vp = V[(size_t)p * n + r], vq = V[(size_t)q * n + r];
                    V[(size_t)p * n + r] = c * vp - s * vq;
                    V[(size_t)q * n + r] = s * vp + c * vq;
                }
            }
            __syncthreads();
        }
    }
    for (int e = tid; e < n * n; e += kJacThreads) Vout[e] = V[e];
    for (int i = tid; i < n; i += kJacThreads) evals[i] = ap[pk_idx(i, i)];
}

// ---------------------------------------------------------------------------
// Grid-wide barrier for a cooperative launch: a monotonic arrival counter;
// barrier number b completes when it reaches (b + 1) * gridDim.x.  The wait is
// bounded (~1 s); on expiry it records kErrWaitTimeout and sets *abort, after
// which every block leaves its loops at the next barrier.
// (skip_arrival: the test hook of amica_test_arm_wait_fault, a block that does
// not arrive, so that the others' waits run out.)
__device__ __forceinline__ bool grid_barrier(unsigned* count, unsigned target, volatile int* abort,
                                             int* err, long long wait_cycles, bool skip_arrival = false) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (!skip_arrival) atomicAdd(count, 1u);
        const long long t0 = clock64();
        while (true) {
            const unsigned v = *(volatile unsigned*)count;
            if (v >= target || *abort) break;
            if (clock64() - t0 > wait_cycles) {
                *abort = 1;
                atomicOr(err, amica::kErrWaitTimeout);
                break;
            }
        }
        __threadfence();
    }
    __syncthreads();
    return *abort == 0;
}

// The Jacobi eigendecomposition of k_jacobi_smem (same round-robin schedule,
// rotation formula, 2 x 2 block transforms, eigenvector update and stopping
// rule) with the packed triangle and V in global memory, rounds spread over all
// blocks of a cooperative launch: every block forms the round's n/2 rotations
// from the packed triangle, a grid barrier, the blocks share out the 2 x 2 block
// and V updates, and a second grid barrier ends the round.  Loads of shared
// state bypass L1.
struct JacGlobal {
    double* ap;        // packed upper triangle, n (n + 1) / 2
    double* part;      // per-block partial sums of the stopping test, 2 per block
    unsigned* count;   // barrier counter (zero at launch)
    int* abort;        // zero at launch
    long long wait_cycles;   // bound of every barrier wait (~1 s)
    int skip_block;          // test hook: this block skips its first arrival (-1: none)
};
__global__ void __launch_bounds__(kJacThreads, 1) k_jacobi_grid(const double* __restrict__ C,
                                                                double* __restrict__ V,
                                                                double* __restrict__ evals, int n,
                                                                JacGlobal g, int* err,
                                                                const int* __restrict__ done) {
    if (*done) return;                                  // the same in every block
    __shared__ double cs[128], sn[128];
    __shared__ int pp[128], qq[128];
    __shared__ double red[32];
    const int tid = threadIdx.x;
    const int gtid = blockIdx.x * kJacThreads + tid, gthreads = gridDim.x * kJacThreads;
    const int np = (n * (n + 1)) / 2;
    const int ne = n + (n & 1), half = ne / 2;
    const int nblk = half * (half + 1) / 2;
    double* ap = g.ap;
    unsigned bar = 0;
    for (int e = gtid; e < n * n; e += gthreads) {
        const int r = e % n, c = e / n;
        if (r <= c) ap[pk_idx(r, c)] = C[e];
        V[e] = (r == c) ? 1.0 : 0.0;
    }
    if (!grid_barrier(g.count, (++bar) * gridDim.x, g.abort, err, g.wait_cycles,
                      (int)blockIdx.x == g.skip_block)) return;
    for (int sweep = 0; sweep < 40; sweep++) {
        double off = 0.0, tot = 0.0;
        for (int e = gtid; e < np; e += gthreads) {
            int j = (int)((sqrt(8.0 * e + 1.0) - 1.0) * 0.5);
            while (pk_idx(0, j + 1) <= e) j++;
            while (pk_idx(0, j) > e) j--;
            const double v = __ldcg(ap + e);
            const bool diag = (e - pk_idx(0, j)) == j;
            tot += diag ? v * v : 2.0 * v * v;
            off += diag ? 0.0 : 2.0 * v * v;
        }
        for (int o = 16; o > 0; o >>= 1) {
            off += __shfl_xor_sync(0xffffffffu, off, o);
            tot += __shfl_xor_sync(0xffffffffu, tot, o);
        }
        if ((tid & 31) == 0) red[tid >> 5] = off;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int w = 0; w < kJacThreads / 32; w++) s += red[w];
            g.part[2 * blockIdx.x] = s;
        }
        __syncthreads();
        if ((tid & 31) == 0) red[tid >> 5] = tot;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int w = 0; w < kJacThreads / 32; w++) s += red[w];
            g.part[2 * blockIdx.x + 1] = s;
        }
        if (!grid_barrier(g.count, (++bar) * gridDim.x, g.abort, err, g.wait_cycles)) return;
        // every block sums the partials in the same order and takes the same decision
        double offt = 0.0, tott = 0.0;
        for (int b = 0; b < (int)gridDim.x; b++) {
            offt += __ldcg(g.part + 2 * b);
            tott += __ldcg(g.part + 2 * b + 1);
        }
        if (offt <= 1e-30 * tott) break;
        // the partials are rewritten next sweep only after every block has read
        // them: the first round's barrier lies in between
        for (int round = 0; round < ne - 1; round++) {
            if (tid < half) {
                auto pos = [&](int j) { return j == 0 ? 0 : 1 + ((j - 1 + round) % (ne - 1)); };
                int p = pos(tid), q = pos(ne - 1 - tid);
                if (p > q) { const int t = p; p = q; q = t; }
                double c = 1.0, s = 0.0;
                if (q < n) {
                    const double apq = __ldcg(ap + pk_idx(p, q));
                    if (fabs(apq) >= 1e-300) {
                        const double app = __ldcg(ap + pk_idx(p, p)), aqq = __ldcg(ap + pk_idx(q, q));
                        const double th = (aqq - app) / (2.0 * apq);
                        const double t = (th >= 0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
                        c = 1.0 / sqrt(t * t + 1.0);
                        s = t * c;
                    }
                }
                pp[tid] = p; qq[tid] = q; cs[tid] = c; sn[tid] = s;
            }
            // every block has read the diagonal entries that the round's K = L
            // blocks are about to overwrite
            if (!grid_barrier(g.count, (++bar) * gridDim.x, g.abort, err, g.wait_cycles)) return;
            // A <- J^T A J: block (K, L), K <= L, numbered column by column
            for (int e = gtid; e < nblk; e += gthreads) {
                int L = (int)((sqrt(8.0 * e + 1.0) - 1.0) * 0.5);
                while ((L + 1) * (L + 2) / 2 <= e) L++;
                while (L * (L + 1) / 2 > e) L--;
                const int K = e - L * (L + 1) / 2;
                const int pK = pp[K], qK = qq[K], pL = pp[L], qL = qq[L];
                const double cK = cs[K], sK = sn[K], cL = cs[L], sL = sn[L];
                if (K == L) {
                    if (qK < n && sK != 0.0) {
                        const double app = __ldcg(ap + pk_idx(pK, pK)), aqq = __ldcg(ap + pk_idx(qK, qK));
                        const double apq = __ldcg(ap + pk_idx(pK, qK));
                        ap[pk_idx(pK, pK)] = cK * cK * app - 2.0 * cK * sK * apq + sK * sK * aqq;
                        ap[pk_idx(qK, qK)] = sK * sK * app + 2.0 * cK * sK * apq + cK * cK * aqq;
                        ap[pk_idx(pK, qK)] = 0.0;
                    }
                    continue;
                }
                if (sK == 0.0 && sL == 0.0) continue;
                const bool hq = qK < n, hqL = qL < n;
                const double b11 = __ldcg(ap + pk_sym(pK, pL));
                const double b12 = hqL ? __ldcg(ap + pk_sym(pK, qL)) : 0.0;
                const double b21 = hq ? __ldcg(ap + pk_sym(qK, pL)) : 0.0;
                const double b22 = (hq && hqL) ? __ldcg(ap + pk_sym(qK, qL)) : 0.0;
                const double d11 = cL * b11 - sL * b12, d12 = sL * b11 + cL * b12;
                const double d21 = cL * b21 - sL * b22, d22 = sL * b21 + cL * b22;
                ap[pk_sym(pK, pL)] = cK * d11 - sK * d21;
                if (hqL) ap[pk_sym(pK, qL)] = cK * d12 - sK * d22;
                if (hq) ap[pk_sym(qK, pL)] = sK * d11 + cK * d21;
                if (hq && hqL) ap[pk_sym(qK, qL)] = sK * d12 + cK * d22;
            }
            // V <- V J, one (rotation, row) pair per work item
            for (int e = gtid; e < half * n; e += gthreads) {
                const int k = e / n, r = e - k * n;
                const int p = pp[k], q = qq[k];
                const double s = sn[k];
                if (q >= n || s == 0.0) continue;
                const double c = cs[k];
                const double vp = __ldcg(V + (size_t)p * n + r), vq = __ldcg(V + (size_t)q * n + r);
                V[(size_t)p * n + r] = c * vp - s * vq;
                V[(size_t)q * n + r] = s * vp + c * vq;
            }
            if (!grid_barrier(g.count, (++bar) * gridDim.x, g.abort, err, g.wait_cycles)) return;
        }
    }
    for (int i = gtid; i < n; i += gthreads) evals[i] = __ldcg(ap + pk_idx(i, i));
}

// x_out[t][i] = sum_k S(i,k) (x[t][k] - mean[k]) in FP64 on the tensor cores
// (mma.sync m8n8k4), rounded once to FP32 (padded channels zero).  A CTA keeps S
// (all of it up to 128 channels; a slice of 64 output channels above, blockIdx.y)
// in shared memory and walks sample tiles; a warp computes 16 samples x 16
// channels, so that two loads of each operand feed four products; both operands
// have a row stride of 4 doubles modulo 16 (fragment loads free of bank
// conflicts).  Stages come as in k_cov_mma.  Bound by the FP64 pipe
// (3.3e10 flop at n = 128, T = 1M, 0.9 ms at 36.7 TFLOP/s; 1.26 ms); the FMA form with 4
// x 4 register blocks took 2.77 ms there, in 128 channels whatever n, and the
// form above 128 channels 690 us at n = 160, T = 50k.
struct SpherePlan {
    int nt, mt, rows, kpad, yslices;   // 16-channel and 16-sample warp tiles, samples per tile, padded K
    int threads;
    size_t smem;
};
SpherePlan sphere_plan(int n) {
    SpherePlan p;
    const int nb = (n + 31) / 32;
    p.kpad = 32 * nb;
    p.nt = n <= 128 ? 2 * nb : 4;
    p.yslices = n <= 128 ? 1 : (n + 63) / 64;
    p.mt = n <= 128 ? 16 / p.nt : 2;                   // 16, 16, 12 and 16 warps; 8 above 128 channels
    for (;; p.mt = 1) {                                // 4 warps above 208 channels
        p.rows = 16 * p.mt;
        p.threads = 32 * p.nt * p.mt;
        p.smem = sizeof(double) * ((size_t)p.kpad * (16 * p.nt + 4) + 2 * (size_t)p.rows * (p.kpad + 4)) +
                 sizeof(float) * (size_t)p.rows * n;
        if (p.mt == 1 || p.smem + 4096 <= 232448) return p;
    }
}
__global__ void __launch_bounds__(512, 1) k_apply_sphere(const float* __restrict__ x, int64_t T, int n,
                                                         const double* __restrict__ mean,
                                                         const double* __restrict__ S, float* __restrict__ xo,
                                                         int ldx, int tf32, int nt, int mt, int kpad, int* err) {
    extern __shared__ __align__(16) double ssm[];
    const int lds = 16 * nt + 4, ldk = kpad + 4, rows = 16 * mt, nb = kpad >> 5;
    double* Ss = ssm;                                  // Ss[k * lds + i] = S(i0 + i, k)
    double* xc = ssm + (size_t)kpad * lds;             // [2] tiles, xc[r * ldk + k]
    float* raw = reinterpret_cast<float*>(xc + 2 * (size_t)rows * ldk);   // [rows][n]
    __shared__ double mean_s[256];
    __shared__ uint64_t bar;
    __shared__ int abort_s;
    volatile int* abort_flag = &abort_s;
    const int tid = threadIdx.x, nthr = blockDim.x, warp = tid >> 5, lane = tid & 31, nw = nthr >> 5;
    const int g = lane >> 2, q = lane & 3;
    const int i0 = 16 * nt * blockIdx.y;
    const int wn = warp % nt, wm = warp / nt;
    const int64_t ntile = (T + rows - 1) / rows;
    if (tid == 0) {
        abort_s = 0;
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (blockIdx.x < ntile) load_run(raw, x, (int64_t)blockIdx.x * rows, T, rows, n, &bar);
    }
    for (int k = warp; k < kpad; k += nw)
        for (int il = lane; il < 16 * nt; il += 32) {
            const int i = i0 + il;
            Ss[k * lds + il] = (i < n && k < n) ? S[(size_t)k * n + i] : 0.0;
        }
    for (int i = tid; i < 256; i += nthr) mean_s[i] = i < n ? mean[i] : 0.0;
    __syncthreads();
    uint32_t stage = 0;
    for (int64_t tile = blockIdx.x; tile < ntile; tile += gridDim.x, stage++) {
        const int64_t t0 = tile * rows;
        double* xb = xc + (size_t)(stage & 1) * rows * ldk;
        mbar_wait(&bar, stage & 1, abort_flag, err);
        each_element(rows, nb, nw, [&](int r, int k) {
            xb[r * ldk + k] = (t0 + r < T && k < n) ? (double)raw[r * n + k] - mean_s[k] : 0.0;
        });
        __syncthreads();
        if (tid == 0 && tile + gridDim.x < ntile) load_run(raw, x, (tile + gridDim.x) * rows, T, rows, n, &bar);
        double acc[2][2][2] = {};
        const double* pa = xb + (16 * wm + g) * ldk + q;
        const double* pb = Ss + q * lds + 16 * wn + g;
        const int ksteps = (n + 3) >> 2;
#pragma unroll 4
        for (int s = 0; s < ksteps; s++) {
            const double a0 = pa[4 * s], a1 = pa[8 * ldk + 4 * s];
            const double b0 = pb[4 * s * lds], b1 = pb[4 * s * lds + 8];
            dmma884(acc[0][0][0], acc[0][0][1], a0, b0);
            dmma884(acc[0][1][0], acc[0][1][1], a0, b1);
            dmma884(acc[1][0][0], acc[1][0][1], a1, b0);
            dmma884(acc[1][1][0], acc[1][1][1], a1, b1);
        }
#pragma unroll
        for (int a = 0; a < 2; a++) {
            const int64_t t = t0 + 16 * wm + 8 * a + g;
            if (t >= T) continue;
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int i = i0 + 16 * wn + 8 * c + 2 * q;   // even, and ldx a multiple of 32
                if (i >= ldx) continue;
                float2 v = make_float2((float)acc[a][c][0], (float)acc[a][c][1]);
                if (tf32) v = make_float2(round_tf32(v.x), round_tf32(v.y));
                *reinterpret_cast<float2*>(xo + t * ldx + i) = v;
            }
        }
        // the last slice also owns the padding channels past it
        if (blockIdx.y + 1 == gridDim.y)
            for (int i = i0 + 16 * nt + 2 * lane; i < ldx; i += 64)
                for (int r = warp; r < rows && t0 + r < T; r += nw)
                    *reinterpret_cast<float2*>(xo + (t0 + r) * ldx + i) = make_float2(0.f, 0.f);
    }
}

__global__ void k_convert(const double* __restrict__ xs, int64_t T, int n, float* __restrict__ xo,
                          int ldx, int tf32) {
    const int64_t total = T * (int64_t)ldx;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = e / ldx;
        const int i = (int)(e % ldx);
        const float v = (i < n) ? (float)xs[t * n + i] : 0.f;
        xo[e] = tf32 ? round_tf32(v) : v;
    }
}

// The preprocessing of one fit in three steps, so that a fit whose samples are
// spread over several contexts can add the sums of every shard between them:
//   pp_colsum:  column sums / div of the raw data;
//   pp_scatter: sum_t (x_t - mean)(x_t - mean)^T / div (do_sphere 1 only);
//   pp_finish:  the eigendecomposition of the covariance, S and ldetS, and
//               the sphered data x = S (raw - mean) in the layout of the E-step.
// evwork: >= 4 n^2 + 4 n doubles.
int sm_count() {
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm;
}

// The steps' scratch: the partial sums and covariances, then the eigensolver's
// state.  A shorter one gives fewer partials and CTAs.
struct Scratch {
    double* p;
    size_t len;   // doubles, at least preprocess_min_ws(n)
};
constexpr int kJacCtas = 64;   // of the cooperative eigensolver

// samples per CTA of the column sums: eight CTAs per SM
int64_t colsum_chunk(int64_t T, int n, size_t len) {
    const int64_t ctas = std::min<int64_t>(8 * (int64_t)sm_count(), (int64_t)(len / n));
    return std::max<int64_t>((T + ctas - 1) / ctas, 64);
}
int cov_ranges(int n, size_t len) {
    return (int)std::min<size_t>(sm_count() / cov_plan(n).ysplit, len / ((size_t)n * n));
}

cudaError_t pp_colsum(const float* raw, int64_t T, int n, double div, Scratch ws, double* out,
                      cudaStream_t st) {
    const int64_t chunk = colsum_chunk(T, n, ws.len);
    const int nblk = (int)((T + chunk - 1) / chunk);
    k_colsum<<<nblk, kSumThreads, 0, st>>>(raw, T, n, chunk, ws.p);
    k_mean<<<(n + 31) / 32, 32 * kFoldWarps, 0, st>>>(ws.p, nblk, n, div, out);
    return cudaGetLastError();
}

cudaError_t pp_scatter(const float* raw, int64_t T, int n, const double* means, double div,
                       Scratch ws, double* out, int* err, cudaStream_t st) {
    const CovPlan p = cov_plan(n);
    // a range is a whole number of stages; ranges past T are empty and leave zeros
    const int ncov = cov_ranges(n, ws.len);
    const int64_t chunk = ((T + ncov - 1) / ncov + p.rows - 1) / p.rows * p.rows;
    cudaError_t e = cudaFuncSetAttribute(k_cov_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem);
    if (e != cudaSuccess) return e;
    k_cov_mma<<<dim3(ncov, p.ysplit), p.threads, p.smem, st>>>(raw, T, n, chunk, means, ws.p, p.nb, p.ntl, p.nrep,
                                                             p.rows, err);
    k_cov_reduce<<<(n * n + 31) / 32, 32 * kFoldWarps, 0, st>>>(ws.p, ncov, n, div, out);
    return cudaGetLastError();
}

// var_ready: evwork's variance slot already holds the do_sphere 2 variances
cudaError_t pp_finish(const float* raw, int64_t T, int n, int do_sphere, const double* means,
                      const double* cov, double* sphere, double* evwork, double* ldetS_dev,
                      float* x, int ldx, int tf32, int* err, Scratch ws, bool var_ready,
                      cudaStream_t st, long long fault_wait_cycles) {
    const bool big = n > 128;
    const int nsm = sm_count();
    cudaError_t e = cudaSuccess;
    double* V = evwork;
    double* ev = evwork + (size_t)n * n;
    double* var = ev + n;
    int* done = reinterpret_cast<int*>(var + n);
    if (do_sphere == 1) {
        // the armed test hook is about the cooperative solver's waits: let it run
        e = fault_wait_cycles > 0 ? cudaMemsetAsync(done, 0, sizeof(int), st)
                                  : amica::launch_eig_cluster(cov, V, ev, n, done, st);
        if (e != cudaSuccess) return e;
    }
    if (do_sphere == 1 && !big) {
        const size_t jsmem = sizeof(double) * (size_t)((((n * (n + 1)) / 2 + 1) & ~1) + n * n);
        e = cudaFuncSetAttribute(k_jacobi_smem, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)jsmem);
        if (e != cudaSuccess) return e;
        k_jacobi_smem<<<1, kJacThreads, jsmem, st>>>(cov, V, ev, n, done);
    } else if (do_sphere == 1) {
        // Jacobi state in the partial buffer: packed triangle, the stopping-test
        // partials, the barrier counter and the abort flag
        int per_sm = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_jacobi_grid, kJacThreads, 0);
        if (e != cudaSuccess || per_sm < 1) return e ? e : cudaErrorInvalidValue;
        const int nb = nsm < kJacCtas ? nsm : kJacCtas;
        const size_t np = (size_t)n * (n + 1) / 2;
        double* part = ws.p;
        JacGlobal jg;
        jg.ap = part;
        jg.part = part + np;
        jg.count = reinterpret_cast<unsigned*>(part + np + 2 * nb);
        jg.abort = reinterpret_cast<int*>(part + np + 2 * nb + 1);
        jg.wait_cycles = fault_wait_cycles > 0 ? fault_wait_cycles : 2000000000LL;
        jg.skip_block = fault_wait_cycles > 0 ? 0 : -1;
        e = cudaMemsetAsync(part + np + 2 * nb, 0, 2 * sizeof(double), st);
        if (e != cudaSuccess) return e;
        double* covp = const_cast<double*>(cov);
        void* args[] = {(void*)&covp, (void*)&V, (void*)&ev, (void*)&n, (void*)&jg, (void*)&err, (void*)&done};
        e = cudaLaunchCooperativeKernel((const void*)k_jacobi_grid, dim3(nb), dim3(kJacThreads), args, 0, st);
        if (e != cudaSuccess) return e;
    } else if (do_sphere == 2 && !var_ready) {
        k_var<<<n, 256, 0, st>>>(raw, T, n, means, var);
    }
    k_sphere<<<(n * n + 255) / 256, 256, 0, st>>>(V, ev, var, n, do_sphere, sphere, ldetS_dev);
    // the scratch is done with: the rows past T, which the kernel below leaves out
    e = cudaMemsetAsync(x + (size_t)T * ldx, 0, sizeof(float) * amica::x_tail_len(ldx), st);
    if (e != cudaSuccess) return e;
    const SpherePlan p = sphere_plan(n);
    e = cudaFuncSetAttribute(k_apply_sphere, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem);
    if (e != cudaSuccess) return e;
    const int64_t ntile = (T + p.rows - 1) / p.rows;
    const int grid = (int)(ntile < nsm / p.yslices ? ntile : nsm / p.yslices);
    k_apply_sphere<<<dim3(grid, p.yslices), p.threads, p.smem, st>>>(raw, T, n, means, sphere, x, ldx, tf32, p.nt,
                                                                   p.mt, p.kpad, err);
    return cudaGetLastError();
}

}  // namespace

namespace amica {

// least scratch (doubles): one partial covariance, or the cooperative
// eigensolver's state
size_t preprocess_min_ws(int n) {
    const size_t nn = (size_t)n * n, jac = (size_t)n * (n + 1) / 2 + 2 * kJacCtas + 2;
    return std::max(nn, jac);
}

// x holds T x ldx + x_tail_len(ldx) floats, and at least 2 preprocess_min_ws(n):
// until the sphered data are written to it, it serves as the scratch; the floats
// past T x ldx are left zero.
// fault_wait_cycles > 0 arms the test hook of amica_test_arm_wait_fault for
// this launch (cooperative eigensolver only: block 0 skips its first arrival,
// every wait is bounded by fault_wait_cycles).
static Scratch x_scratch(float* x, int64_t T, int n, int ldx) {
    return Scratch{reinterpret_cast<double*>(x), std::max((size_t)T * ldx / 2, preprocess_min_ws(n))};
}
cudaError_t launch_preprocess(const float* raw, int64_t T, int n, int do_sphere, double* means,
                              double* cov, double* sphere, double* evwork, double* ldetS_dev,
                              float* x, int ldx, int tf32, int* err, cudaStream_t st,
                              long long fault_wait_cycles) {
    if (n > 256 || ldx > 256) return cudaErrorInvalidValue;
    const Scratch ws = x_scratch(x, T, n, ldx);
    cudaError_t e = pp_colsum(raw, T, n, (double)T, ws, means, st);
    if (e == cudaSuccess && do_sphere == 1) e = pp_scatter(raw, T, n, means, (double)T, ws, cov, err, st);
    if (e == cudaSuccess)
        e = pp_finish(raw, T, n, do_sphere, means, cov, sphere, evwork, ldetS_dev, x, ldx, tf32, err, ws,
                      false, st, fault_wait_cycles);
    return e;
}

// Sharded preprocessing: the column sums of this shard's raw data (n doubles).
// (x may be in use: the scratch is its own.)
cudaError_t launch_shard_colsum(const float* raw, int64_t T, int n, double* sums, cudaStream_t st) {
    if (n > 256) return cudaErrorInvalidValue;
    Scratch ws{nullptr, (size_t)8 * sm_count() * n};
    cudaError_t e = cudaMallocAsync(&ws.p, sizeof(double) * ws.len, st);
    if (e != cudaSuccess) return e;
    e = pp_colsum(raw, T, n, 1.0, ws, sums, st);
    cudaFreeAsync(ws.p, st);
    return e;
}

// means = sums / T_total (the column sums of all shards), then the scatter of
// this shard's raw data about them, n x n doubles.
cudaError_t launch_shard_scatter(const float* raw, int64_t T, int n, const double* sums, int64_t T_total,
                                 double* means, double* scatter, int* err, cudaStream_t st) {
    if (n > 256 || T_total < 1) return cudaErrorInvalidValue;
    Scratch ws{nullptr, (size_t)sm_count() * n * n};
    cudaError_t e = cudaMallocAsync(&ws.p, sizeof(double) * ws.len, st);
    if (e != cudaSuccess) return e;
    k_mean<<<(n + 31) / 32, 32 * kFoldWarps, 0, st>>>(sums, 1, n, (double)T_total, means);
    e = pp_scatter(raw, T, n, means, 1.0, ws, scatter, err, st);
    cudaFreeAsync(ws.p, st);
    return e;
}

// S and ldetS from the scatter of all shards (T_total samples; do_sphere 1 and
// 2 read it, 0 ignores it), applied to this shard's samples.  x as in
// launch_preprocess.
cudaError_t launch_shard_finish(const float* raw, int64_t T, int n, int do_sphere, const double* means,
                                const double* scatter, int64_t T_total, double* cov, double* sphere,
                                double* evwork, double* ldetS_dev, float* x, int ldx, int tf32, int* err,
                                cudaStream_t st) {
    if (n > 256 || ldx > 256 || T_total < 2) return cudaErrorInvalidValue;
    if (do_sphere != 0)
        k_scale_scatter<<<(n * n + 255) / 256, 256, 0, st>>>(scatter, n, (double)T_total, cov,
                                                             evwork + (size_t)n * n + n);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
        e = pp_finish(raw, T, n, do_sphere, means, cov, sphere, evwork, ldetS_dev, x, ldx, tf32, err,
                      x_scratch(x, T, n, ldx), true, st, 0);
    return e;
}

cudaError_t launch_convert_sphered(const double* xs, int64_t T, int n, float* x, int ldx, int tf32,
                                   cudaStream_t st) {
    k_convert<<<2048, 256, 0, st>>>(xs, T, n, x, ldx, tf32);
    const cudaError_t e = cudaGetLastError();
    // a sphering that ended with an error may have left scratch past T
    return e != cudaSuccess ? e : cudaMemsetAsync(x + (size_t)T * ldx, 0, sizeof(float) * x_tail_len(ldx), st);
}

}  // namespace amica
