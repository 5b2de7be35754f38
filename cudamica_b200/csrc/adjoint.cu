// Hand-written adjoint of the AMICA log-likelihood.
//
// L = sum_t P(t),  P(t) = log sum_h exp(Lt_h(t)),
// Lt_h(t) = log gm_h + log|det W_h| + ldetS + sum_i log sum_j exp(Q_hij(t)),
// Q = log alpha + 0.5 log beta - log 2 - lgamma(1 + 1/rho) - |y|^rho,
// y = sqrt(beta) (b - mu),  b = W_h (x_t - c_h)
// (the density of src/kernels.cu:282-307 and the likelihood of :317-450).
//
// With u = v_h z_hij = dP/dQ and f' = rho sign(y) |y|^(rho-1):
//   dL/dmu   = sqrt(beta) sum u f'
//   dL/dbeta = (sum u - sum u f' y) / (2 beta)
//   dL/drho  = sum u psi(1 + 1/rho) / rho^2 - sum u |y|^rho log|y|^rho / rho
//   dL/dW_h  = (sum v_h) W_h^{-T} - (sum g (x - c_h)^T),  g = sum_j sqrt(beta) u f'
// Every sum is one the fused E-step already forms per tile (it recomputes the
// responsibilities from b and never stores the M*m*n*T posterior), so the
// adjoint sweep IS the E-step kernel run in gradient mode, followed by this
// FP64 finalisation.  The natural-gradient direction the M-step uses,
// I - phi, equals (dL/dW_h) W_h^T / vsum_h.
#include <cmath>

#include "common.cuh"

namespace amica {
cudaError_t launch_estep_plain(const EStepArgs& a, int NP, int nclusters, cudaStream_t st);
cudaError_t launch_estep_tc(const EStepArgs& a, int NP, int nclusters, cudaStream_t st, int split, int shape);
// mstep.cu
cudaError_t launch_reduce(const double* partial, double* raw, int nslots, int M, int n, int m, int psi_step,
                          cudaStream_t st);
cudaError_t launch_adjoint_dw(const double* raw, const double* A, double* out, int n, int m, int M,
                              cudaStream_t st);
}

using namespace amica;

namespace {

__device__ double psi_dev(double x) {
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

// out: [0] sum P (relative), then dW (M n n, column-major), dmu, dbeta, drho
// (M m n).  blockIdx.y = model; dW here only where the n x n block is
// Psi = sum g x^T (sum g (x - c)^T = Psi - gsum c^T); where it is phi, dW is a
// product with A and comes from launch_adjoint_dw.
__global__ void __launch_bounds__(256) k_adjoint_finalize(const double* __restrict__ raw, const double* __restrict__ A,
                                   const double* __restrict__ c, const double* __restrict__ beta,
                                   const double* __restrict__ rho, double* __restrict__ out, int n,
                                   int m, int M, int psi_is_phi) {
    const int h = blockIdx.y;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    PartLayout PL{n, m};
    const double* R = raw + (size_t)h * PL.stride();
    const double vsum = R[1];
    if (h == 0 && t0 == 0) out[0] = R[0];
    if (!psi_is_phi) {
        double* dW = out + 1 + (size_t)h * n * n;
        const double* Ah = A + (size_t)h * n * n;
        const double* Psi = R + PL.psi();
        const double* gs = R + PL.gs();
        for (int e = t0; e < n * n; e += nt) {
            const int i = e % n, k = e / n;   // dW(i,k) stored at k*n + i; W^{-T}(i,k) = A(k,i)
            dW[e] = vsum * Ah[(size_t)i * n + k] - (Psi[(size_t)k * n + i] - gs[i] * c[(size_t)h * n + k]);
        }
    }
    const size_t off_mu = 1 + (size_t)M * n * n;
    const size_t mnM = (size_t)M * m * n;
    for (int e = t0; e < m * n; e += nt) {
        const size_t idx = (size_t)h * m * n + e;
        const double bt = beta[idx], r = rho[idx];
        const double us = R[PL.mix(kUs) + e];
        out[off_mu + idx] = sqrt(bt) * R[PL.mix(kMn) + e];
        out[off_mu + mnM + idx] = (us - R[PL.mix(kBd) + e]) / (2.0 * bt);
        out[off_mu + 2 * mnM + idx] = us * psi_dev(1.0 + 1.0 / r) / (r * r) - R[PL.mix(kRn) + e] / r;
    }
}

}  // namespace

namespace amica {

// The adjoint sweep: the fused E-step in gradient mode into `partial`.
cudaError_t launch_adjoint(const EStepArgs& a0, int NP, double* grad_partial, int nclusters,
                           cudaStream_t st, bool use_tc, int tc_shape) {
    EStepArgs a = a0;
    a.grad_mode = 1;
    a.update_rho = 1;
    a.partial = grad_partial;
    a.split_phi = nullptr;   // the gradient sweep does not need phi's split correction
    return use_tc ? launch_estep_tc(a, NP, nclusters, st, 0, tc_shape) : launch_estep_plain(a, NP, nclusters, st);
}

// The product phi A^T runs as the M-step's tiled FP64 GEMM: with one CTA per
// model walking it entry by entry this step took 333 us at n = 100, M = 2, and
// the slot sum with one thread per entry 98 us.
cudaError_t launch_adjoint_finalize(const double* grad_partial, double* raw, int nslots, int psi_step, int n,
                                    int m, int M, const double* A, const double* c,
                                    const double* beta, const double* rho, double* out,
                                    int psi_is_phi, cudaStream_t st) {
    cudaError_t e = launch_reduce(grad_partial, raw, nslots, M, n, m, psi_step, st);
    if (e != cudaSuccess) return e;
    const int len = psi_is_phi ? m * n : n * n;
    k_adjoint_finalize<<<dim3((len + 255) / 256, M), 256, 0, st>>>(raw, A, c, beta, rho, out, n, m, M, psi_is_phi);
    e = cudaGetLastError();
    if (e != cudaSuccess || !psi_is_phi) return e;
    return launch_adjoint_dw(raw, A, out + 1, n, m, M, st);
}

}  // namespace amica
