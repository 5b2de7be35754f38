// Eigendecomposition C = V diag(d) V^T of the channel covariance for the
// sphering (replaces MAGMA's dsyevd in src/preprocess.cu:126-229), n <= 256, on
// one thread-block cluster of up to 8 CTAs (16 above 192 channels).
//
//   1. C = L L^T, blocked Cholesky.
//   2. One-sided Jacobi on the columns of L (Hestenes rotations; applied to the
//      Cholesky factor as in Veselic and Hari, "A note on a one-sided Jacobi
//      algorithm", 1989): rotating pairs of columns until all are orthogonal
//      gives L J = V diag(sqrt(d)), so that the eigenvectors are the normalised
//      columns, d their squared norms, and no second matrix is accumulated.
//
// Columns are dealt to 2K blocks of b (K CTAs).  A CTA holds two blocks; it
// rotates the b^2 cross pairs in b steps, warp w keeping column w of the top
// block in registers while the bottom block's columns go round the warps
// through shared memory, then sends both blocks on to their next CTA (the
// round-robin schedule on blocks) through distributed shared memory: one cluster
// barrier per 2K - 1 block rounds of a sweep, and within a CTA one barrier per b
// rotations.  Bound by the latency of a step (dot product, rotation, update):
// the whole matrix is a few KB per warp and the FP64 pipe is mostly idle, so the
// split aims at few pairs per warp (one) and a short chain per pair.  The
// two-sided form that it replaced re-read the matrix and the eigenvectors from
// one SM's shared memory (n = 128: 5.2 ms) or, above 128 channels, from L2 with
// two grid barriers per round (n = 160: 15.9 ms).
//
// A covariance that is not numerically positive definite (a pivot below
// n eps max diag: rank-deficient data) is left to that form: *done stays 0.  So is
// a device that has no 16 SMs for one cluster.
#include <cooperative_groups.h>
#include <cstdint>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int kMaxCtas = 16;       // above 8: the non-portable cluster size
constexpr int kMaxBlk = 12;        // columns per block (n = 192 on 8 CTAs)
constexpr int kMaxSweeps = 40;

__device__ __forceinline__ double rcp_approx(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}
__device__ __forceinline__ double rsqrt_approx(double x) {
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The rotation that makes two columns of squared norms a, b and inner product c
// orthogonal.  The tangent needs only a few digits (what it misses is left of c
// for the next sweep); cosine and sine come from it with cos^2 + sin^2 = 1 to
// the last bits: 1/sqrt(1 + t^2) by two Newton steps from a 20-bit start.
__device__ __forceinline__ void rotation(double a, double b, double c, double& cs, double& sn, double& t) {
    const double z = (b - a) * (0.5 * rcp_approx(c));
    const double w = fma(z, z, 1.0);
    t = copysign(rcp_approx(fabs(z) + w * rsqrt_approx(w)), z);
    const double q = fma(t, t, 1.0), hq = 0.5 * q;
    double r = rsqrt_approx(q);
    r = r * fma(-hq * r, r, 1.5);
    r = r * fma(-hq * r, r, 1.5);
    cs = r;
    sn = t * r;
}

template <int NE>
__global__ void __launch_bounds__(32 * kMaxBlk, 1)
    k_eig_cluster(const double* __restrict__ C, double* __restrict__ V, double* __restrict__ evals, int n, int b,
                  int* __restrict__ done) {
    constexpr int LD = 32 * NE;
    extern __shared__ __align__(16) double esm[];      // [2 sets][top, bottom][b][LD]
    __shared__ double nrm[2 * kMaxBlk];
    __shared__ int flags[2][kMaxCtas], fail[kMaxCtas];
    cg::cluster_group cluster = cg::this_cluster();
    const int K = (int)cluster.num_blocks(), me = (int)cluster.block_rank();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto col = [&](int set, int tb, int j) -> double* { return esm + (size_t)((set * 2 + tb) * b + j) * LD; };

    // ---- this warp's columns of C (lower triangle) and the largest diagonal entry
    double x[2][NE];                                   // top and bottom column
#pragma unroll
    for (int tb = 0; tb < 2; tb++) {
        const int c = (tb * K + me) * b + w;
#pragma unroll
        for (int e = 0; e < NE; e++) {
            const int r = lane + 32 * e;
            x[tb][e] = (c < n && r < n && r >= c) ? C[(size_t)c * n + r] : 0.0;
        }
    }
    double dmax = 0.0;
    for (int i = lane; i < n; i += 32) dmax = fmax(dmax, C[(size_t)i * n + i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
    const double eps = 2.220446049250313e-16;
    const double piv_min = (double)n * eps * dmax;
    if (threadIdx.x < kMaxCtas) fail[threadIdx.x] = 0;
    int bad = 0;
    cluster.sync();                                    // every CTA is running before remote stores
    // ---- Cholesky by panels of b columns: the owner sweeps a panel and sends
    // it to every CTA (sets 0 and 1 of the column buffers' top halves in turn),
    // which apply it to their later columns
    for (int p = 0; p < 2 * K; p++) {
        const int owner = p % K, tbp = p / K, k0 = p * b, buf = p & 1;
        if (k0 >= n) break;                            // the same in every CTA
        if (me == owner) {
            for (int t = 0; t < b && k0 + t < n; t++) {
                const int k = k0 + t;
                if (w == t) {
                    double d = 0.0;
#pragma unroll
                    for (int e = 0; e < NE; e++)
                        if (e == (k >> 5)) d = __shfl_sync(0xffffffffu, tbp ? x[1][e] : x[0][e], k & 31);
                    const bool ok = d > piv_min;       // false for NaN
                    if (!ok) bad = 1;
                    const double inv = ok ? 1.0 / sqrt(d) : 0.0;
#pragma unroll
                    for (int e = 0; e < NE; e++) {
                        const double v = (tbp ? x[1][e] : x[0][e]) * inv;
                        if (tbp) x[1][e] = v; else x[0][e] = v;
                        for (int q = 0; q < K; q++) cluster.map_shared_rank(col(buf, 0, t), q)[lane + 32 * e] = v;
                    }
                }
                __syncthreads();
                const int c = k0 + w;
                if (w > t && c < n) {
                    const double* pc = col(buf, 0, t);
                    const double l = pc[c];
#pragma unroll
                    for (int e = 0; e < NE; e++) {
                        const int r = lane + 32 * e;
                        const double u = r >= c ? l * pc[r] : 0.0;
                        if (tbp) x[1][e] -= u; else x[0][e] -= u;
                    }
                }
            }
        }
        cluster.sync();                                // panel p is in every CTA
        const int np = min(b, n - k0);
#pragma unroll
        for (int tb = 0; tb < 2; tb++) {
            const int blk = tb * K + me, c = blk * b + w;
            if (blk > p && c < n) {
                for (int t = 0; t < np; t++) {
                    const double* pc = col(buf, 0, t);
                    const double l = pc[c];
#pragma unroll
                    for (int e = 0; e < NE; e++) {
                        const int r = lane + 32 * e;
                        if (r >= c) x[tb][e] = fma(-l, pc[r], x[tb][e]);
                    }
                }
            }
        }
    }
    if (bad && lane == 0)
        for (int q = 0; q < K; q++) cluster.map_shared_rank(fail, q)[me] = 1;
    cluster.sync();                                    // panels read, failures known
    for (int q = 0; q < K; q++) bad |= fail[q];
    if (bad) return;                                   // the same in every CTA; no remote access follows

    // ---- one-sided Jacobi
#pragma unroll
    for (int e = 0; e < NE; e++) {
        col(0, 0, w)[lane + 32 * e] = x[0][e];
        col(0, 1, w)[lane + 32 * e] = x[1][e];
    }
    const double tol2 = 4.0 * n * eps * eps;           // (2 sqrt(n) eps)^2
    // a sweep that met no inner product above this (relative) leaves ones of the
    // order of its square
    const double more2 = 1e-22;
    const int be = b + (b & 1);
    int cur = 0, rotated = 0;
    // one pair, p and q in registers; true if they were rotated
    auto pair = [&](double* p, double* q, double a, double bb, double& t, double& c) -> bool {
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int e = 0; e < NE; e += 2) {
            s0 = fma(p[e], q[e], s0);
            if (e + 1 < NE) s1 = fma(p[e + 1], q[e + 1], s1);
        }
        c = warp_sum(s0 + s1);
        const double c2 = c * c, ab = a * bb;
        if (!(c2 > tol2 * ab)) return false;
        if (c2 > more2 * ab) rotated = 1;
        double cs, sn;
        rotation(a, bb, c, cs, sn, t);
#pragma unroll
        for (int e = 0; e < NE; e++) {
            const double u = p[e], v = q[e];
            p[e] = fma(cs, u, -sn * v);
            q[e] = fma(sn, u, cs * v);
        }
        return true;
    };
    auto norm2 = [&](const double* v) -> double {
        double s = 0.0;
#pragma unroll
        for (int e = 0; e < NE; e++) s = fma(v[e], v[e], s);
        return warp_sum(s);
    };
    __syncthreads();
    for (int sweep = 0; sweep < kMaxSweeps; sweep++) {
        rotated = 0;
        double t, c;
        // the pairs inside each block, once per sweep: be/2 pairs of the
        // round-robin schedule per block and step
        for (int step = 0; step < be - 1; step++) {
            for (int idx = w; idx < be; idx += b) {
                const int tb = idx >= be / 2, pr = idx - tb * (be / 2);
                auto pos = [&](int j) { return j == 0 ? 0 : 1 + (j - 1 + step) % (be - 1); };
                const int i0 = pos(pr), i1 = pos(be - 1 - pr);
                if (i0 < b && i1 < b) {
                    double *cp = col(cur, tb, i0), *cq = col(cur, tb, i1);
                    double p[NE], q[NE];
#pragma unroll
                    for (int e = 0; e < NE; e++) { p[e] = cp[lane + 32 * e]; q[e] = cq[lane + 32 * e]; }
                    if (pair(p, q, norm2(p), norm2(q), t, c)) {
#pragma unroll
                        for (int e = 0; e < NE; e++) { cp[lane + 32 * e] = p[e]; cq[lane + 32 * e] = q[e]; }
                    }
                }
            }
            __syncthreads();
        }
        for (int br = 0; br < 2 * K - 1; br++) {
            double p[NE], q[NE];
#pragma unroll
            for (int e = 0; e < NE; e++) { p[e] = col(cur, 0, w)[lane + 32 * e]; q[e] = col(cur, 1, w)[lane + 32 * e]; }
            double a = norm2(p);
            double bb = norm2(q);
            int j = w;
            for (int r = 0; r < b; r++) {
                if (pair(p, q, a, bb, t, c)) {
                    a = fma(-t, c, a);
                    bb = fma(t, c, bb);
                }
                if (r + 1 == b) break;
                // pass the bottom column on: warp w takes column j + 1 next
                double* cq = col(cur, 1, j);
#pragma unroll
                for (int e = 0; e < NE; e++) cq[lane + 32 * e] = q[e];
                if (lane == 0) nrm[j] = bb;
                __syncthreads();
                j = j + 1 == b ? 0 : j + 1;
                cq = col(cur, 1, j);
#pragma unroll
                for (int e = 0; e < NE; e++) q[e] = cq[lane + 32 * e];
                bb = nrm[j];
                // (a column is overwritten only by the warp that has it)
            }
            // both blocks to their next CTA, other set
            const int tq = K == 1 || me == 0 ? me : (me < K - 1 ? me + 1 : K - 1);
            const int ttb = K > 1 && me == K - 1 ? 1 : 0;
            const int bq = K == 1 ? 0 : (me > 0 ? me - 1 : 1);
            const int btb = K == 1 || me > 0 ? 1 : 0;
            double* dt = cluster.map_shared_rank(col(cur ^ 1, ttb, w), tq);
            double* db = cluster.map_shared_rank(col(cur ^ 1, btb, j), bq);
#pragma unroll
            for (int e = 0; e < NE; e++) { dt[lane + 32 * e] = p[e]; db[lane + 32 * e] = q[e]; }
            if (br == 2 * K - 2) {
                const int any = __syncthreads_or(rotated);
                if (threadIdx.x < K) cluster.map_shared_rank(flags[sweep & 1], threadIdx.x)[me] = any;
            }
            cluster.sync();
            cur ^= 1;
        }
        int any = 0;
        for (int q = 0; q < K; q++) any |= flags[sweep & 1][q];
        if (!any) break;                               // the same in every CTA
    }
    // a whole sweep returns every block to where it began
#pragma unroll
    for (int tb = 0; tb < 2; tb++) {
        const int c = (tb * K + me) * b + w;
        if (c < n) {
            double v[NE];
#pragma unroll
            for (int e = 0; e < NE; e++) v[e] = col(cur, tb, w)[lane + 32 * e];
            const double d = norm2(v), inv = 1.0 / sqrt(d);
#pragma unroll
            for (int e = 0; e < NE; e++)
                if (lane + 32 * e < n) V[(size_t)c * n + lane + 32 * e] = v[e] * inv;
            if (lane == 0) evals[c] = d;
        }
    }
    if (me == 0 && threadIdx.x == 0) *done = 1;
}

template <int NE>
cudaError_t launch_eig(const double* C, double* V, double* evals, int n, int K, int b, int* done, cudaStream_t st) {
    const size_t smem = sizeof(double) * 4 * (size_t)b * 32 * NE;
    auto kern = k_eig_cluster<NE>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(K);
    cfg.blockDim = dim3(32 * b);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = K;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (K > 8) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        int fits = 0;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&fits, kern, &cfg);
        if (e != cudaSuccess || fits < 1) {            // *done is 0
            cudaGetLastError();
            return cudaSuccess;
        }
    }
    return cudaLaunchKernelEx(&cfg, kern, C, V, evals, n, b, done);
}

}  // namespace

namespace amica {

// V (n x n, column-major) and evals of the covariance C; *done = 1 when they
// were written, 0 when C is not numerically positive definite.  The cluster has
// as many CTAs as keep 5 to 8 columns in a block (9 to 12 at 129 to 192 channels): a
// step's pairs then run one per warp with two or three warps per scheduler (16 CTAs
// against 8: n = 256 2.2 ms against 2.8, n = 160 the same).
cudaError_t launch_eig_cluster(const double* C, double* V, double* evals, int n, int* done, cudaStream_t st) {
    if (n < 2 || n > 256) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(done, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    const int K = n <= 16 ? 1 : n <= 32 ? 2 : n <= 64 ? 4 : n <= 192 ? 8 : kMaxCtas;
    const int b = (n + 2 * K - 1) / (2 * K);
    switch ((n + 31) / 32) {
        case 1: return launch_eig<1>(C, V, evals, n, K, b, done, st);
        case 2: return launch_eig<2>(C, V, evals, n, K, b, done, st);
        case 3: return launch_eig<3>(C, V, evals, n, K, b, done, st);
        case 4: return launch_eig<4>(C, V, evals, n, K, b, done, st);
        case 5: return launch_eig<5>(C, V, evals, n, K, b, done, st);
        case 6: return launch_eig<6>(C, V, evals, n, K, b, done, st);
        case 7: return launch_eig<7>(C, V, evals, n, K, b, done, st);
        default: return launch_eig<8>(C, V, evals, n, K, b, done, st);
    }
}

}  // namespace amica
