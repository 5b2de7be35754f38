// Kernels of the single-model tensor-core E-step (estep_tc_one.cuh): one fit,
// and the persistent cohort launch over many fits.
#include "estep_tc_one.cuh"

namespace {

__device__ __forceinline__ void named_bar(int id, int nthreads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
__device__ __forceinline__ uint32_t one_tmem_alloc(uint8_t* sm, uint32_t off_misc, bool alloc_warp) {
    uint32_t* holder = (uint32_t*)(sm + off_misc);
    if (alloc_warp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(holder)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    return *holder;
}
__device__ __forceinline__ void one_tmem_free(uint32_t tmem, bool alloc_warp) {
    tc_fence_before();
    __syncthreads();
    if (alloc_warp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// Persistent: CTA c runs tiles c, c + nclusters, ...
template <int MM, int R, int WG, int NST>
__global__ void __launch_bounds__(TcCfg<WG, NST>::kThreads, 1)
    estep_tc_one_kernel(const __grid_constant__ CUtensorMap xmap, EStepArgs a) {
    using Cf = TcCfg<WG, NST>;
    using Sh = OneShape<Cf>;
    if (a.split_phi != nullptr && *a.split_phi != 0) return;   // the split-correction form runs instead
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* sm = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* bar = (uint64_t*)(sm + Sh::OFF_BAR);
    volatile int* abort_flag = (volatile int*)(sm + Sh::OFF_MISC + 8);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cid = blockIdx.x;
    const int ntl = (a.ntiles > cid) ? (a.ntiles - cid + a.nclusters - 1) / a.nclusters : 0;
    if (tid == 0) {
        *abort_flag = 0;
        one_barriers<Cf>(bar, false);
    }
    const uint32_t tmem = one_tmem_alloc(sm, Sh::OFF_MISC, warp == Cf::kDensWarps);
    if (warp < Cf::kDensWarps) one_load_w<Cf>(a.Wf, 128 / R, tmem, warp, lane);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp >= Cf::kDensWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cf::kCtlRegs));
        if (warp == Cf::kDensWarps && lane == 0 && ntl > 0)
            one_control<Cf>(sm, bar, abort_flag, a.err, &xmap, tmem, cid, a.nclusters, ntl);
        __syncwarp();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Cf::kDensRegs));
        one_density<MM, R, Cf>(sm, bar, abort_flag, a, tmem, warp, lane, cid, a.nclusters, ntl, cid);
    }
    one_tmem_free(tmem, warp == Cf::kDensWarps);
}

// ---------------------------------------------------------------- cohort
// One persistent launch over the sample tiles of many single-model fits of the
// same m (a cohort of subjects with their own channel counts and lengths).  A
// work item is a run of consecutive tiles of one subject; CTA c processes items
// item_off[c] .. item_off[c + 1] - 1 in order.  Per item the density warps load
// the subject's W into tensor memory while the control thread re-arms the
// barriers; each item's statistics go to its own partial-slot group of the
// subject.
template <int MM>
using CohortCfg = TcCfg<(MM >= 4 ? 2 : 3), 2>;        // tc_default_shape
template <int MM>
__global__ void __launch_bounds__(CohortCfg<MM>::kThreads, 1)
    estep_tc_cohort_kernel(const TcCohortSub* __restrict__ subs, const CUtensorMap* __restrict__ maps,
                           const TcCohortItem* __restrict__ items, const int* __restrict__ item_off) {
    using Cf = CohortCfg<MM>;
    constexpr int kThreads = Cf::kThreads, kDensWarps = Cf::kDensWarps;
    constexpr int kCtlRegs = Cf::kCtlRegs, kDensRegs = Cf::kDensRegs;
    using Sh = OneShape<Cf>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* sm = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* bar = (uint64_t*)(sm + Sh::OFF_BAR);
    volatile int* abort_flag = (volatile int*)(sm + Sh::OFF_MISC + 8);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int i0 = item_off[blockIdx.x], i1 = item_off[blockIdx.x + 1];
    if (tid == 0) *abort_flag = 0;
    const uint32_t tmem = one_tmem_alloc(sm, Sh::OFF_MISC, warp == kDensWarps);
    if (warp >= kDensWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kCtlRegs));
        for (int ii = i0; ii < i1; ii++) {
            const TcCohortItem itm = items[ii];
            if (tid == kDensWarps * 32) one_barriers<Cf>(bar, ii > i0);
            tc_fence_before();
            named_bar(1, kThreads);                   // item set up
            tc_fence_after();
            if (warp == kDensWarps && lane == 0 && itm.ntiles > 0)
                one_control<Cf>(sm, bar, abort_flag, subs[itm.sub].a.err, maps + itm.sub, tmem, itm.tile0, 1,
                                itm.ntiles);
            __syncwarp();
            tc_fence_before();
            named_bar(2, kThreads);                   // item done
            tc_fence_after();
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kDensRegs));
        for (int ii = i0; ii < i1; ii++) {
            const TcCohortItem itm = items[ii];
            const TcCohortSub& S = subs[itm.sub];
            one_load_w<Cf>(S.a.Wf, 128 / S.R, tmem, warp, lane);
            tc_fence_before();
            named_bar(1, kThreads);
            tc_fence_after();
            if (S.R == 4)
                one_density<MM, 4, Cf>(sm, bar, abort_flag, S.a, tmem, warp, lane, itm.tile0, 1, itm.ntiles, itm.slot);
            else if (S.R == 2)
                one_density<MM, 2, Cf>(sm, bar, abort_flag, S.a, tmem, warp, lane, itm.tile0, 1, itm.ntiles, itm.slot);
            else
                one_density<MM, 1, Cf>(sm, bar, abort_flag, S.a, tmem, warp, lane, itm.tile0, 1, itm.ntiles, itm.slot);
            tc_fence_before();
            named_bar(2, kThreads);
            tc_fence_after();
        }
    }
    one_tmem_free(tmem, warp == kDensWarps);
}

// ---------------------------------------------------------------- host side
template <class K>
cudaError_t one_prepare(K kern, size_t smem, int threads, int split_regs) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    // setmaxnreg draws on the registers the block is launched with (launch_tc)
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, kern);
    if (e != cudaSuccess) return e;
    return fa.numRegs * threads < split_regs ? cudaErrorInvalidConfiguration : cudaSuccess;
}

template <int MM, int R, int WG, int NST>
cudaError_t launch_one(const EStepArgs& a, int nclusters, cudaStream_t st) {
    using Cf = TcCfg<WG, NST>;
    using Sh = OneShape<Cf>;
    constexpr int kS = Cf::kS;
    PFN_encodeTiled enc = get_encode();
    if (!enc) return cudaErrorNotSupported;
    if (a.ldx * R != 128 || a.M != 1) return cudaErrorInvalidValue;
    const int64_t rows = (a.T + R - 1) / R;
    if (a.ntiles != (int)((rows + kS - 1) / kS)) return cudaErrorInvalidValue;
    CUtensorMap map;
    cuuint64_t dims[2] = {128, (cuuint64_t)rows};
    cuuint64_t strides[1] = {128 * 4};
    cuuint32_t box[2] = {32, (cuuint32_t)kS};
    cuuint32_t estr[2] = {1, 1};
    if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)a.x, dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    auto kern = estep_tc_one_kernel<MM, R, WG, NST>;
    const size_t smem = Sh::BYTES + 1024;
    cudaError_t e = one_prepare(kern, smem, Cf::kThreads, WG * 128 * Cf::kDensRegs + 128 * Cf::kCtlRegs);
    if (e != cudaSuccess) return e;
    kern<<<nclusters, Cf::kThreads, smem, st>>>(map, a);
    return cudaGetLastError();
}

template <int WG, int NST>
cudaError_t launch_one_shape(const EStepArgs& a, int nclusters, cudaStream_t st) {
    const int R = tc_pack(a.n);
#define AMICA_ONE_CASE(MMV) \
    if (a.m == MMV) return R == 1 ? launch_one<MMV, 1, WG, NST>(a, nclusters, st) \
                                  : (R == 2 ? launch_one<MMV, 2, WG, NST>(a, nclusters, st) \
                                            : launch_one<MMV, 4, WG, NST>(a, nclusters, st));
    AMICA_ONE_CASE(1) AMICA_ONE_CASE(2) AMICA_ONE_CASE(3) AMICA_ONE_CASE(4) AMICA_ONE_CASE(5)
#undef AMICA_ONE_CASE
    return cudaErrorInvalidValue;
}

template <int MM>
cudaError_t launch_cohort(const TcCohortSub* subs, const CUtensorMap* maps, const TcCohortItem* items,
                          const int* item_off, int nctas, cudaStream_t st) {
    auto kern = estep_tc_cohort_kernel<MM>;
    using Cf = CohortCfg<MM>;
    const size_t smem = OneShape<Cf>::BYTES + 1024;
    cudaError_t e = one_prepare(kern, smem, Cf::kThreads, Cf::kWG * 128 * Cf::kDensRegs + 128 * Cf::kCtlRegs);
    if (e != cudaSuccess) return e;
    kern<<<nctas, Cf::kThreads, smem, st>>>(subs, maps, items, item_off);
    return cudaGetLastError();
}

}  // namespace

namespace amica {

// The plain form (no split correction of phi) at M = 1 in a tile shape: density
// warpgroups and x stages as in TcCfg.
cudaError_t launch_estep_tc_one(const EStepArgs& a, int nclusters, cudaStream_t st, int shape) {
    switch (shape) {
        case 0: return launch_one_shape<3, 2>(a, nclusters, st);
        case 1: return launch_one_shape<2, 2>(a, nclusters, st);
        case 2: return launch_one_shape<2, 3>(a, nclusters, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_estep_tc_cohort(const TcCohortSub* subs, const void* maps, const TcCohortItem* items,
                                   const int* item_off, int nctas, int m, cudaStream_t st) {
    const CUtensorMap* mp = (const CUtensorMap*)maps;
    switch (m) {
        case 1: return launch_cohort<1>(subs, mp, items, item_off, nctas, st);
        case 2: return launch_cohort<2>(subs, mp, items, item_off, nctas, st);
        case 3: return launch_cohort<3>(subs, mp, items, item_off, nctas, st);
        case 4: return launch_cohort<4>(subs, mp, items, item_off, nctas, st);
        case 5: return launch_cohort<5>(subs, mp, items, item_off, nctas, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace amica
