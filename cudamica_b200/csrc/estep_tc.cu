// The mixed-precision fused E-step (estep_tc.cuh) in its default shape of 3
// density warpgroups, the tensor-core self-test and the host interface that
// picks a shape and a form.
#include "estep_tc.cuh"

namespace {

// ---------------------------------------------------------------- self-test
// One CTA runs a single contraction D[128][N] = A[128][K] . B[N][K]^T with the
// layouts, descriptors and TMEM access of the E-step kernel (B K-major in
// shared memory, as the x tile in MMA1 and the b tile in MMA2):
//   mode 0: A = tf32(A) K-major in shared memory (W_hi, G)
//   mode 1: A = tf32(A) in tensor memory (the A-from-TMEM form of W_lo)
//   mode 2: A = hi + lo split, hi in shared memory, lo in tensor memory (MMA1)
// K is a multiple of 16 (<= 64); N a multiple of 16 (<= 128).
__global__ void __launch_bounds__(128, 1) umma_selftest_kernel(const float* __restrict__ A,
                                                               const float* __restrict__ B,
                                                               float* __restrict__ D, int mode,
                                                               int N, int K, int* err) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* sm = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* As = sm;                      // K-major, 128 rows, ceil(K/32) blocks of 16 KB
    uint8_t* Bs = sm + 2 * 16384;          // K-major, N rows
    uint64_t* bar = (uint64_t*)(sm + 2 * 16384 + 2 * 16384);
    uint32_t* holder = (uint32_t*)(bar + 2);
    volatile int* abort_flag = (volatile int*)(bar + 3);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int e = tid; e < 128 * K; e += 128) {
        const int r = e / K, c = e % K;
        *(float*)(As + sw128_off(r, c, 128)) = tf32_rna(A[e]);
    }
    for (int e = tid; e < N * K; e += 128) {
        const int r = e / K, c = e % K;
        *(float*)(Bs + sw128_off(r, c, N)) = tf32_rna(B[e]);
    }
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(holder)), "r"(128u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *holder;                     // D: columns [0, N); A in TMEM: [N, N+K)
    if (mode >= 1) {
        const int r = warp * 32 + lane;
        for (int k0 = 0; k0 < K; k0 += 16) {
            float v[16];
            for (int q = 0; q < 16; q++) {
                const float w = A[(size_t)r * K + k0 + q];
                v[q] = mode == 1 ? tf32_rna(w) : tf32_rna(w - tf32_rna(w));
            }
            tmem_st16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(N + k0), v);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (tid == 0) {
        const uint32_t abase = smem_u32(As), bbase = smem_u32(Bs);
        const uint32_t id = idesc_tf32(128, N, 0, 0);
        for (int kk = 0; kk < K / 8; kk++) {
            const uint64_t bd = sdesc(bbase + (kk >> 2) * N * 128 + (kk & 3) * 32, 16, 1024);
            if (mode == 0 || mode == 2) {
                const uint64_t ad = sdesc(abase + (kk >> 2) * 128 * 128 + (kk & 3) * 32, 16, 1024);
                tc_mma_tf32(tmem, ad, bd, id, kk > 0 ? 1u : 0u);
            }
            if (mode >= 1)
                tc_mma_tf32_ta(tmem, tmem + (uint32_t)(N + kk * 8), bd, id,
                               (mode == 2 || kk > 0) ? 1u : 0u);
        }
        tc_commit(&bar[0]);
    }
    __syncwarp();
    const bool ok = mbar_wait(&bar[0], 0u, abort_flag, err);
    tc_fence_after();
    if (ok) {
        for (int c0 = 0; c0 < N; c0 += 16) {
            float v[16];
            tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
            for (int q = 0; q < 16; q++) D[(size_t)(warp * 32 + lane) * N + c0 + q] = v[q];
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(128u)
                     : "memory");
    }
}
}  // namespace

namespace amica {

int tc_selftest(int mode, int N, int K, const float* hA, const float* hB, float* hD, int* derr) {
    if (mode < 0 || mode > 2 || N % 16 || N < 16 || N > 64 || K % 16 || K < 16 || K > 64)
        return -3;
    float *dA, *dB, *dD;
    int* err;
    if (cudaMalloc(&dA, sizeof(float) * 128 * K) != cudaSuccess) return -1;
    cudaMalloc(&dB, sizeof(float) * N * K);
    cudaMalloc(&dD, sizeof(float) * 128 * N);
    cudaMalloc(&err, sizeof(int));
    cudaMemset(err, 0, sizeof(int));
    cudaMemcpy(dA, hA, sizeof(float) * 128 * K, cudaMemcpyHostToDevice);
    cudaMemcpy(dB, hB, sizeof(float) * N * K, cudaMemcpyHostToDevice);
    const int smem = 4 * 16384 + 1024 + 64;
    cudaFuncSetAttribute(umma_selftest_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    umma_selftest_kernel<<<1, 128, smem>>>(dA, dB, dD, mode, N, K, err);
    cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess) {
        cudaMemcpy(hD, dD, sizeof(float) * 128 * N, cudaMemcpyDeviceToHost);
        cudaMemcpy(derr, err, sizeof(int), cudaMemcpyDeviceToHost);
    }
    cudaFree(dA); cudaFree(dB); cudaFree(dD); cudaFree(err);
    return e == cudaSuccess ? 0 : -20;
}

// Tile shapes the context can run (TcCfg): 0 = 3 density warpgroups,
// 48-sample tiles, 2 x stages; 1 = 2 warpgroups, 32-sample tiles, 2 stages; 2 = 2
// warpgroups, 3 stages.
cudaError_t launch_estep_tc_one(const EStepArgs& a, int nclusters, cudaStream_t st, int shape);
int tc_wg2_max_clusters(int n, int m, int M, int nst);
cudaError_t tc_wg2_launch(const EStepArgs& a, int nclusters, cudaStream_t st, int split, int nst);

int tc_num_shapes() { return 3; }
// The shape of a new context whose configuration names none, and of the cohort
// kernel.  With one model and four or five mixtures the single-phase kernel's sums
// and parameters take about 170 registers a thread, more than 3 density warpgroups
// leave (136): 2 warpgroups measured 168 us against 282 at n = 64, T = 300k, m = 5,
// 150 against 153 at m = 4 (n = 32: 72 against 78; n = 128: 287 against 285).  With several
// models and five mixtures the log2|y| cache fits beside 2 warpgroups only: 1.12 ms
// against 1.17 at n = 128, T = 400k, M = 2 at the start of a fit and 0.95 against 0.97 in
// the middle; at M = 3, T = 300k 1.41 against 1.43 and 1.12 against 1.09 (m = 4 the other
// way: 1.00 against 0.92 and 0.85 against 0.76 at M = 2).
int tc_default_shape(int m, int M) { return m == 5 || (M == 1 && m == 4) ? 1 : 0; }
static int shape_wg(int shape) { return shape == 0 ? 3 : 2; }
// Samples per tile: 16 rows per warpgroup, R samples per row.
int tc_tile_samples(int n, int shape) { return 16 * shape_wg(shape) * tc_pack(n); }
// Partial slots per cluster, and the stride between the slots that carry phi.
int tc_partial_groups(int n, int shape) { return shape_wg(shape) * tc_pack(n); }
int tc_psi_step(int shape) { return shape_wg(shape); }

int tc_supported(int n, int m, int M) {
    return n >= 2 && n <= 128 && m >= 1 && m <= 5 && M >= 1 && M <= kMaxModels;
}

// Every channel count runs the 128-lane kernel (packed below 65 channels).
int tc_max_clusters(int n, int m, int M, int shape) {
    if (!tc_supported(n, m, M) || shape < 0 || shape >= tc_num_shapes()) return -1;
    if (shape == 0) return tc_max_clusters_shape<3, 2>(n, m, M);
    return tc_wg2_max_clusters(n, m, M, shape == 1 ? 2 : 3);
}

// The x tensor map of one subject for the cohort kernel (a.x read as rows of
// 128 floats, R samples each); `map` receives a CUtensorMap (128 bytes).
int tc_cohort_encode_map(const EStepArgs& a, void* map) {
    PFN_encodeTiled enc = get_encode();
    if (!enc) return -1;
    const int R = tc_pack(a.n);
    if (a.ldx * R != 128) return -1;
    const int64_t rows = (a.T + R - 1) / R;
    cuuint64_t dims[2] = {(cuuint64_t)128, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)128 * 4};
    cuuint32_t box[2] = {32, (cuuint32_t)(tc_tile_samples(a.n, tc_default_shape(a.m, 1)) / R)};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc((CUtensorMap*)map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)a.x, dims, strides, box,
                     estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : -1;
}

// CTAs of the cohort launch: one per SM.
int tc_cohort_ctas() {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm;
}

// split as in launch_tc_shape.  With one model the plain form is the single-phase
// kernel of estep_tc_one.cuh.
cudaError_t launch_estep_tc(const EStepArgs& a, int NP, int nclusters, cudaStream_t st, int split, int shape) {
    if (NP != tc_np(a.n) || a.ldx != NP) return cudaErrorInvalidValue;
    if (a.M == 1 && split != 1) {
        const cudaError_t e = launch_estep_tc_one(a, nclusters, st, shape);
        if (e != cudaSuccess || split == 0) return e;
        split = 1;
    }
    if (shape == 0) return launch_tc_shape<3, 2>(a, nclusters, st, split);
    if (shape == 1 || shape == 2) return tc_wg2_launch(a, nclusters, st, split, shape == 1 ? 2 : 3);
    return cudaErrorInvalidValue;
}

}  // namespace amica
