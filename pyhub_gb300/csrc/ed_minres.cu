// ed_minres.cu -- MINRES on the complement of a ground state.
//
// (H - E0) x = b with b projected off psi, the adjoint solve of the density
// matrix gradient (no reference counterpart: the reference has no
// derivatives).  Paige and Saunders, SIAM J. Numer. Anal. 12, 1975: three-term
// Lanczos recurrence, Givens rotations of its tridiagonal, work vectors only;
// every operator application is projected onto the complement of psi.
//
// An iteration is the H*v, two vector passes and two scalar kernels, with its
// scalars on the device: as separate vector operations it was ~24 launches,
// a dozen passes over memory and two host synchronisations.
//   pass 1   the previous iteration's w and x, and four sums
//   scalars  a1 = <psi, r>, alpha
//   pass 2   p = r - a1 psi - beta v_prev - alpha v (over v_prev), |p|^2
//   scalars  the rotation, the coefficients of w and x, the stop test
// with r = H v - E0 v.  Lanczos vectors are stored unnormalised, their scales
// among the scalars.  Bound by the launches on small sectors, by the FP64 pipe
// (15 operations per element beside the H*v's ~25) on large ones.
// Differentiable step of 10 sites (63,504 states, 67 iterations): 32.4 -> 14.9 ms.
#include "ed_common.cuh"

#include <algorithm>
#include <cmath>

namespace ed {

// device scalars
enum {
    kMSv, kMSp, kMBeta, kMA1, kMAlpha, kMDbar, kMEps, kMCs, kMSn, kMPhibar, kMTol, kMDone, kMIters, kMBeta1,
    kMPend, kMOldEps, kMDelta, kMIGamma, kMPhi, kMScal = 32
};

constexpr int kMrThreads = 256;

__device__ __forceinline__ void put_sums(double (&s)[4], double *__restrict__ part, int n)
{
    __shared__ double red[kMrThreads / 32][4];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        s[q] = warp_sum(s[q]);
        if (lane == 0) red[warp][q] = s[q];
    }
    __syncthreads();
    if (threadIdx.x < n) {
        double t = 0.0;
        for (int w = 0; w < kMrThreads / 32; ++w) t += red[w][threadIdx.x];
        part[(int64_t)threadIdx.x * gridDim.x + blockIdx.x] = t;
    }
}

// sums of psi.b (start of the solve)
__global__ void __launch_bounds__(kMrThreads) minres_dot_kernel(int64_t n, const double *__restrict__ a,
                                                                const double *__restrict__ b, double *__restrict__ part)
{
    double s[4] = {0, 0, 0, 0};
    for (int64_t i = (int64_t)blockIdx.x * kMrThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kMrThreads)
        s[0] = fma(a[i], b[i], s[0]);
    put_sums(s, part, 1);
}

// out = b - a1 psi (out may be b), partial |out|^2
__global__ void __launch_bounds__(kMrThreads) minres_project_kernel(int64_t n, const double *b,
                                                                    const double *__restrict__ psi, double *out,
                                                                    const double *__restrict__ S,
                                                                    double *__restrict__ part)
{
    const double a1 = S[kMA1];
    double s[4] = {0, 0, 0, 0};
    for (int64_t i = (int64_t)blockIdx.x * kMrThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kMrThreads) {
        const double v = fma(-a1, psi[i], b[i]);
        out[i] = v;
        s[0] = fma(v, v, s[0]);
    }
    put_sums(s, part, 1);
}

// w1 <- (v_prev - oldeps w1 - delta w) / gamma, x += phi w1 (when an iteration left them pending), and
// with SUMS: psi.r, v.r, v.psi, v.v_prev of the unscaled vectors, r = q - E0 v.
template <bool SUMS>
__global__ void __launch_bounds__(kMrThreads) minres_pass1_kernel(int64_t n, double e0, const double *__restrict__ q,
                                                                  const double *__restrict__ v,
                                                                  const double *__restrict__ vp,
                                                                  const double *__restrict__ psi,
                                                                  const double *__restrict__ w, double *__restrict__ w1,
                                                                  double *__restrict__ x, const double *__restrict__ S,
                                                                  double *__restrict__ part)
{
    const bool pend = S[kMPend] != 0.0, done = S[kMDone] != 0.0;
    if (done && !pend) return;
    const double sp = S[kMSp], oe = S[kMOldEps], de = S[kMDelta], ig = S[kMIGamma], phi = S[kMPhi];
    double s[4] = {0, 0, 0, 0};
    for (int64_t i = (int64_t)blockIdx.x * kMrThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kMrThreads) {
        const double p = vp[i];
        if (pend) {
            const double t = fma(-de, w[i], fma(-oe, w1[i], sp * p)) * ig;
            w1[i] = t;
            x[i] = fma(phi, t, x[i]);
        }
        if (SUMS && !done) {
            const double u = v[i], r = fma(-e0, u, q[i]), f = psi[i];
            s[0] = fma(f, r, s[0]);
            s[1] = fma(u, r, s[1]);
            s[2] = fma(u, f, s[2]);
            s[3] = fma(u, p, s[3]);
        }
    }
    if (SUMS && !done) put_sums(s, part, 4);
}

__global__ void __launch_bounds__(kMrThreads) minres_pass2_kernel(int64_t n, double e0, const double *__restrict__ q,
                                                                  const double *__restrict__ v,
                                                                  const double *__restrict__ psi,
                                                                  double *__restrict__ vp, const double *__restrict__ S,
                                                                  double *__restrict__ part)
{
    if (S[kMDone] != 0.0) return;
    const double sv = S[kMSv], a1 = S[kMA1], bp = S[kMBeta] * S[kMSp], av = S[kMAlpha] * sv + sv * e0;
    double s[4] = {0, 0, 0, 0};
    for (int64_t i = (int64_t)blockIdx.x * kMrThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kMrThreads) {
        const double t = fma(-av, v[i], fma(-bp, vp[i], fma(-a1, psi[i], sv * q[i])));
        vp[i] = t;
        s[0] = fma(t, t, s[0]);
    }
    put_sums(s, part, 1);
}

// The scalars after a pass: mode 0 a1 = psi.b; 1 the start (beta_1 = |v|); 2 after pass 1; 3 after pass 2.
__global__ void __launch_bounds__(256) minres_scalar_kernel(const double *__restrict__ part, int rows, int mode,
                                                            double rtol, double *__restrict__ S)
{
    __shared__ double red[8];
    if (mode >= 2 && S[kMDone] != 0.0) {
        if (threadIdx.x == 0) S[kMPend] = 0.0;
        return;
    }
    double d[4] = {0, 0, 0, 0};
    const int ns = (mode == 2) ? 4 : 1;
    for (int q = 0; q < ns; ++q) {
        d[q] = sum_rows_cta(part + (int64_t)q * rows, rows, 1, red);
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    if (mode == 0) {
        S[kMA1] = d[0];
    } else if (mode == 1) {
        const double b1 = sqrt(d[0]);
        S[kMBeta1] = b1;
        S[kMPhibar] = b1;
        S[kMTol] = rtol * b1;
        S[kMSv] = b1 == 0.0 ? 0.0 : 1.0 / b1;
        S[kMSp] = 0.0;
        S[kMBeta] = 0.0;
        S[kMDbar] = S[kMEps] = S[kMSn] = 0.0;
        S[kMCs] = -1.0;
        S[kMDone] = b1 == 0.0 ? 1.0 : 0.0;
        S[kMIters] = 0.0;
        S[kMPend] = 0.0;
    } else if (mode == 2) {
        const double sv = S[kMSv], a1 = sv * d[0];
        S[kMA1] = a1;
        S[kMAlpha] = sv * sv * d[1] - a1 * sv * d[2] - S[kMBeta] * sv * S[kMSp] * d[3];
        S[kMPend] = 0.0;
    } else {
        const double alpha = S[kMAlpha], bn = sqrt(d[0]);
        const double cs = S[kMCs], sn = S[kMSn], dbar = S[kMDbar], oldeps = S[kMEps];
        const double delta = cs * dbar + sn * alpha, gbar = sn * dbar - cs * alpha;
        S[kMEps] = sn * bn;
        S[kMDbar] = -cs * bn;
        const double gamma = hypot(gbar, bn);
        S[kMIters] += 1.0;
        if (gamma == 0.0) {     // a zero pivot ends the run without this iteration's update
            S[kMDone] = 1.0;
            return;
        }
        const double c1 = gbar / gamma, s1 = bn / gamma, phibar = S[kMPhibar];
        S[kMCs] = c1;
        S[kMSn] = s1;
        S[kMPhi] = c1 * phibar;
        S[kMPhibar] = s1 * phibar;
        S[kMOldEps] = oldeps;
        S[kMDelta] = delta;
        S[kMIGamma] = 1.0 / gamma;
        S[kMPend] = 1.0;
        S[kMSp] = S[kMSv];        // the vectors change roles: v is v_prev of the next iteration
        S[kMSv] = bn == 0.0 ? 0.0 : 1.0 / bn;
        S[kMBeta] = bn;
        if (fabs(s1 * phibar) <= S[kMTol] || bn == 0.0) S[kMDone] = 1.0;
    }
}

static int64_t minres_len(const ed_sector *s, int64_t ld)
{
    return ((s->kind == ED_HUBBARD ? s->nsdn * ld : s->dim) + 31) / 32 * 32;
}

static int minres_grid(int64_t n)
{
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + kMrThreads - 1) / kMrThreads, (int64_t)num_sms() * 4));
}

}  // namespace ed

using namespace ed;

extern "C" int64_t ed_minres_scratch_bytes(const ed_sector *s, int64_t ld)
{
    if (!s) return -1;
    // q, two Lanczos vectors, w and w1; the scalars; the partial sums
    return (5 * minres_len(s, ld) + kMScal + 4 * (int64_t)num_sms() * 4) * (int64_t)sizeof(double) + 256;
}

extern "C" int ed_minres(ed_sector *s, void *stream, int64_t ld, const double *psi, double e0, const double *b, double *x,
                         int maxiter, double rtol, int *iters, double *relres, void *scratch, int64_t scratch_bytes)
{
    clear_error();
    ED_REQUIRE(s != nullptr, "sector is NULL");
    ED_REQUIRE(psi != nullptr && b != nullptr && x != nullptr && iters != nullptr && relres != nullptr, "NULL argument");
    ED_REQUIRE(s->kind != ED_HUBBARD || ld >= s->nsup, "ld=%lld below nsup=%lld", (long long)ld, (long long)s->nsup);
    ED_REQUIRE(scratch != nullptr && scratch_bytes >= ed_minres_scratch_bytes(s, ld),
               "scratch of %lld bytes is below the %lld needed", (long long)scratch_bytes,
               (long long)ed_minres_scratch_bytes(s, ld));
    ED_REQUIRE((reinterpret_cast<uintptr_t>(scratch) % 16) == 0, "scratch must be 16-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    *iters = 0;
    *relres = 0.0;
    const int64_t n = s->kind == ED_HUBBARD ? s->nsdn * ld : s->dim, nv = minres_len(s, ld);
    if (n == 0) return ED_OK;
    // x is cleared before b is read and written while psi and the scratch are in use
    auto apart = [](const void *a, int64_t na, const void *c, int64_t nc) {
        const uintptr_t pa = reinterpret_cast<uintptr_t>(a), pc = reinterpret_cast<uintptr_t>(c);
        return pa + (uintptr_t)na <= pc || pc + (uintptr_t)nc <= pa;
    };
    const int64_t vb = n * (int64_t)sizeof(double), sb = ed_minres_scratch_bytes(s, ld);
    ED_REQUIRE(apart(x, vb, b, vb) && apart(x, vb, psi, vb), "x must not alias b or psi");
    ED_REQUIRE(apart(scratch, sb, x, vb) && apart(scratch, sb, b, vb) && apart(scratch, sb, psi, vb),
               "the scratch must not alias x, b or psi");
    double *q = static_cast<double *>(scratch);
    double *u[2] = {q + nv, q + 2 * nv}, *w[2] = {q + 3 * nv, q + 4 * nv};
    double *S = q + 5 * nv, *part = S + kMScal;
    const int grid = minres_grid(n);
    ED_CHECK_CUDA(cudaMemsetAsync(scratch, 0, sizeof(double) * (size_t)(5 * nv + kMScal), st));   // row padding stays zero
    ED_CHECK_CUDA(cudaMemsetAsync(x, 0, sizeof(double) * (size_t)n, st));
    minres_dot_kernel<<<grid, kMrThreads, 0, st>>>(n, psi, b, part);
    minres_scalar_kernel<<<1, 256, 0, st>>>(part, grid, 0, rtol, S);
    minres_project_kernel<<<grid, kMrThreads, 0, st>>>(n, b, psi, u[0], S, part);
    minres_scalar_kernel<<<1, 256, 0, st>>>(part, grid, 1, rtol, S);
    ED_CHECK_LAUNCH();
    // the host looks after every `chunk` iterations (a finished run's launches return at once): about
    // a million elements' worth of work between looks
    const int chunk = (int)std::max<int64_t>(1, std::min<int64_t>(16, ((int64_t)1 << 20) / n));
    double h[kMScal];
    int it = 0;
    for (;;) {
        const int end = std::min(maxiter, it + chunk);
        for (; it < end; ++it) {
            double *v = u[it & 1], *vp = u[(it + 1) & 1];
            const int rc = ed_hv(s, stream, ED_F64, ld, v, q, 1.0, nullptr, nullptr, 0);
            if (rc) return rc;
            // w of iteration it-1 replaces w1, the one before it
            minres_pass1_kernel<true><<<grid, kMrThreads, 0, st>>>(n, e0, q, v, vp, psi, w[it & 1], w[(it + 1) & 1], x,
                                                                   S, part);
            minres_scalar_kernel<<<1, 256, 0, st>>>(part, grid, 2, rtol, S);
            minres_pass2_kernel<<<grid, kMrThreads, 0, st>>>(n, e0, q, v, psi, vp, S, part);
            minres_scalar_kernel<<<1, 256, 0, st>>>(part, grid, 3, rtol, S);
            ED_CHECK_LAUNCH();
        }
        ED_CHECK_CUDA(cudaMemcpyAsync(h, S, sizeof(h), cudaMemcpyDeviceToHost, st));
        ED_CHECK_CUDA(cudaStreamSynchronize(st));
        if (h[kMDone] != 0.0 || it >= maxiter) break;
    }
    *iters = (int)h[kMIters];
    *relres = h[kMBeta1] == 0.0 ? 0.0 : std::abs(h[kMPhibar]) / h[kMBeta1];
    // the last iteration's x, unless a later pass 1 has applied it; then x off psi
    if (h[kMPend] != 0.0)
        minres_pass1_kernel<false><<<grid, kMrThreads, 0, st>>>(n, e0, q, u[it & 1], u[(it + 1) & 1], psi, w[it & 1],
                                                                w[(it + 1) & 1], x, S, part);
    minres_dot_kernel<<<grid, kMrThreads, 0, st>>>(n, psi, x, part);
    minres_scalar_kernel<<<1, 256, 0, st>>>(part, grid, 0, rtol, S);
    minres_project_kernel<<<grid, kMrThreads, 0, st>>>(n, x, psi, x, S, part);
    ED_CHECK_LAUNCH();
    ED_CHECK_CUDA(cudaStreamSynchronize(st));      // x is final and the scratch free when the call returns
    return ED_OK;
}
