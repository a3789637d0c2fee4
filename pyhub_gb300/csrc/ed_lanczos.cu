// ed_lanczos.cu -- the scalar work of a full-reorthogonalisation Lanczos step,
// kept on the device so that a step enqueues without a host synchronisation.
//
// The reference's LANCZOS (lanczos.f90:50-58) forms alpha_k and beta_k from
// two dot products on the host.  The engine's step also projects H v_k on
// every stored basis vector (delayed classical Gram-Schmidt with the exact
// Gram matrix G of the stored, rounded basis):
//   w = H u_k                                   (ed_hv, unscaled)
//   a_j = <u_j, w>, b_j = <u_j, u_k>            (ed_multidot, one pass)
//   g_j = s_j s_k b_j     (row k of G, v_j = s_j u_j the normalised vectors)
//   c_j = s_j s_k a_j     (= <v_j, H v_k>)
//   y = G^{-1} c,  coef_j = y_j s_j
//   u_{k+1} = s_k w - sum_j coef_j u_j          (ed_update_wscaled)
//   beta_k = ||u_{k+1}||,  s_{k+1} = 1 / beta_k,  alpha_k = c_k.
// G is solved through its inverse Cholesky factor Linv (G = L L^T), grown by
// one row per step: with l = Linv g[0:k] and lam = sqrt(g_k - l.l),
//   Linv[k][0:k] = -(l^T Linv) / lam,  Linv[k][k] = 1 / lam,
// and y = Linv^T (Linv c).  G is within rounding of the identity, so the
// explicit inverse is as accurate as the triangular solves it replaces.
#include "ed_common.cuh"

#include <cooperative_groups.h>

namespace ed {

namespace cg = cooperative_groups;

constexpr int kCoefThreads = 256;
constexpr int kCoefCtas = 8;         // one thread-block cluster
constexpr int kLanczosMax = 8192;    // largest step count a state can hold

// State layout (FP64): [0] stop code, [1] largest |G - I| entry seen,
// [2 .. 2+mmax] scales s_j, then Linv as (mmax+1) x (mmax+1) row-major, then
// four spare vectors of mmax+1 entries.
__host__ __device__ inline int64_t lz_linv_off(int mmax) { return 3 + (int64_t)mmax; }
__host__ __device__ inline int64_t lz_work_off(int mmax) { return lz_linv_off(mmax) + (int64_t)(mmax + 1) * (mmax + 1); }

// Rows of Linv that a CTA of the cluster owns, i = kCoefCtas p + rank: p below this (32 rows at a time).
__host__ __device__ inline int coef_rows(int k) { return (k + 32 * kCoefCtas - 1) / (32 * kCoefCtas) * 32; }
__host__ __device__ inline size_t coef_smem(int k) { return sizeof(double) * (2 * (size_t)(k + 1) + 2 * (size_t)coef_rows(k)); }

// Sum q of the multi-dot, or of its partial rows (the pairing of launch_reduce's warp sum).
__device__ __forceinline__ double dot_sum(const double *__restrict__ dots, int drows, int m, int q)
{
    if (drows == 1) return dots[q];
    double v[kCoefDotRows];
#pragma unroll
    for (int r = 0; r < kCoefDotRows; ++r) v[r] = (r < drows) ? dots[(int64_t)r * m + q] : 0.0;
#pragma unroll
    for (int o = kCoefDotRows / 2; o >= 1; o >>= 1)
#pragma unroll
        for (int r = 0; r < o; ++r) v[r] += v[r + o];
    return v[0];
}

// Part 1 of a step (below): s_k and the stop code from nrm2 = ||u_k||^2, beta_{k-1} through beta when not NULL.
__device__ __forceinline__ void step_scale(int k, double nrm2, const double *__restrict__ state,
                                           const double *__restrict__ alpha, double *__restrict__ beta, double &sk,
                                           double &stop)
{
    stop = state[0];
    sk = state[2 + k];
    if (k < 1 || stop != 0.0) return;
    const double pos = fmax(nrm2, 0.0), bk = sqrt(pos);
    if (!isfinite(nrm2)) {
        stop = -(double)k;
        sk = 0.0;
        return;
    }
    if (beta) beta[k - 1] = bk;
    if (bk <= 1e-13 * fmax(1.0, fabs(alpha[k - 1]))) {
        stop = (double)k;
        sk = 0.0;
    } else {
        sk = rsqrt(pos);
    }
}

// A closing call is part 1 alone: one warp, no cluster to bring up (k = 1 to 8,000: 2.4 us, in the kernel below 2.8).
__global__ void __launch_bounds__(32) lanczos_close_kernel(int k, const double *__restrict__ nrm, double *state,
                                                           const double *__restrict__ alpha, double *__restrict__ beta)
{
    if (threadIdx.x != 0) return;
    double sk, stop;
    step_scale(k, k >= 1 ? nrm[0] : 0.0, state, alpha, beta, sk, stop);
    state[2 + k] = sk;
    if (stop != 0.0) state[0] = stop;
}

// One cluster of kCoefCtas CTAs.  Part 1 (every call, k >= 1): beta_{k-1} and s_k from nrm, with
// the breakdown test of the host loop (beta <= 1e-13 max(1, |alpha|)).
// Part 1 is idempotent: a second call for the same k with the same nrm writes
// the same beta_{k-1} and s_k.  The host's look-ahead relies on it (a run that
// stops at a check has already enqueued the next step, whose part 1 rewrites
// them before the Ritz vector is formed).  Part 2
// (not in a closing call): G row k, Linv row k, coef and alpha_k; it also stops the run
// when u_k is numerically dependent on the basis.  Once stopped, coef is
// written as zeros (and s stays 0), so the vectors that follow are zero and
// finite until the host sees the stop code.
//
// What bounds it: latency.  A dependent FP64 operation takes tens of clocks here, a square root or a
// quotient hundreds, and one SM does 2 FP64 multiply-adds per clock (k^2 / 2 per product with Linv).
// Linv is therefore read twice instead of four times (g and c go through the row pass together, l
// and z through the column pass: the new row's product with c is (c_k - l.z) / lam), its rows are
// dealt over the CTAs of a cluster, whose sums meet once in distributed shared memory, and the
// chain holds no sum over a whole CTA and no quotient.  One CTA with four passes took 12.2,
// 19.2, 33.6 and 72.4 us at k = 10, 40, 100 and 200 (launch included); this form 7.9, 9.2, 10.8 and 13.9.
__global__ void __cluster_dims__(kCoefCtas, 1, 1) __launch_bounds__(kCoefThreads)
    lanczos_coef_kernel(int k, int mmax, const double *__restrict__ dots, int drows, const double *__restrict__ nrm,
                        int nrows, double *state, double *__restrict__ coef, double *__restrict__ alpha,
                        double *__restrict__ beta)
{
    extern __shared__ double dyn[];
    __shared__ double red[8];
    __shared__ double head[2];                       // s_k, stop code
    __shared__ double part[2][kCoefThreads / 32];    // per warp: l.l and l.z over the CTA's rows
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), t = threadIdx.x, lane = t & 31;
    double *s = state + 2;
    // ||u_k||^2, or its partial sums in the order of launch_reduce
    double nrm2 = 0.0;
    if (nrows > 64) {
        nrm2 = sum_rows_cta(nrm, nrows, 1, red);
    } else if (nrows > 1) {
        if (t < 32) {
            for (int b = t; b < nrows; b += 32) nrm2 += nrm[b];
            nrm2 = warp_sum(nrm2);
        }
    } else if (k >= 1) {
        nrm2 = nrm[0];
    }
    if (t == 0) {
        double sk, stop;
        step_scale(k, nrm2, state, alpha, rank == 0 ? beta : nullptr, sk, stop);
        head[0] = sk;
        head[1] = stop;
    }
    __syncthreads();
    const double sk = head[0], stop = head[1];
    if (stop != 0.0) {
        cluster.sync();      // every CTA has read the state before rank 0 writes it
        if (rank != 0) return;
        if (t == 0) {
            s[k] = sk;
            state[0] = stop;
        }
        for (int j = t; j <= k; j += kCoefThreads) coef[j] = 0.0;
        return;
    }
    double *Linv = state + lz_linv_off(mmax);
    const int64_t ldl = mmax + 1;
    double *g = dyn, *c = g + (k + 1);       // Gram row and projections; then this CTA's column sums
    double *l = c + (k + 1), *z = l + coef_rows(k);   // Linv g and Linv c on the CTA's rows
    long long off = 0;     // bits of the largest |G - I| entry: non-negative doubles order as integers
    for (int j = t; j <= k; j += kCoefThreads) {
        const double f = (j == k ? sk : s[j]) * sk;
        const double gj = f * dot_sum(dots, drows, 2 * (k + 1), k + 1 + j);
        g[j] = gj;
        c[j] = f * dot_sum(dots, drows, 2 * (k + 1), j);
        off = max(off, __double_as_longlong(fabs(j == k ? gj - 1.0 : gj)));
    }
    __syncthreads();
    const double gk = g[k], ck = c[k];
    // l = Linv[0:k][0:k] g, z = Linv[0:k][0:k] c on the CTA's rows: 8 lanes per row
    const int sub = t >> 3, l8 = t & 7;
    double ll = 0.0, lz = 0.0;
    for (int p = sub; p < coef_rows(k); p += 32) {
        const int i = p * kCoefCtas + rank;
        double tg = 0.0, tc = 0.0;
        if (i < k) {
            const double *row = Linv + (int64_t)i * ldl;
#pragma unroll 4
            for (int j = l8; j <= i; j += 8) {
                const double v = row[j];
                tg = fma(v, g[j], tg);
                tc = fma(v, c[j], tc);
            }
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            tg += __shfl_xor_sync(0xffffffffu, tg, o);
            tc += __shfl_xor_sync(0xffffffffu, tc, o);
        }
        if (l8 == 0) {
            l[p] = tg;
            z[p] = tc;
        }
        ll = fma(tg, tg, ll);
        lz = fma(tg, tc, lz);
    }
#pragma unroll
    for (int o = 8; o <= 16; o <<= 1) {      // the eight lanes of a row hold the same sums
        ll += __shfl_xor_sync(0xffffffffu, ll, o);
        lz += __shfl_xor_sync(0xffffffffu, lz, o);
    }
    if (lane == 0) {
        part[0][t >> 5] = ll;
        part[1][t >> 5] = lz;
    }
    __syncthreads();       // l and z are written, g and c are read
    // column sums over the CTA's rows
    for (int j = t; j < k; j += kCoefThreads) {
        double a = 0.0, b = 0.0;
#pragma unroll 4
        for (int p = (max(j - rank, 0) + kCoefCtas - 1) / kCoefCtas; p * kCoefCtas + rank < k; ++p) {
            const double v = Linv[(int64_t)(p * kCoefCtas + rank) * ldl + j];
            a = fma(v, l[p], a);
            b = fma(v, z[p], b);
        }
        g[j] = a;
        c[j] = b;
    }
    cluster.sync();
    // l.l and l.z over the cluster, by every warp: kCoefCtas x 8 warps' sums, two per lane
    {
        constexpr int NW = kCoefThreads / 32;
        static_assert(kCoefCtas * NW == 64, "two partial sums per lane");
        const double *p0 = cluster.map_shared_rank(&part[0][0], lane / NW);
        const double *p1 = cluster.map_shared_rank(&part[0][0], lane / NW + 32 / NW);
        ll = warp_sum(p0[lane % NW] + p1[lane % NW]);
        lz = warp_sum(p0[NW + lane % NW] + p1[NW + lane % NW]);
    }
    // a healthy step has lam^2 = g_k - |l|^2 within rounding of 1; below g_k / 2 the stored
    // vector lies mostly inside the span of the basis (a Krylov space exhausted to rounding
    // noise): the run stops with k steps, before the inverse factor would blow up
    if (k >= 1 && !(gk - ll >= 0.5 * gk)) {
        if (rank == 0) {
            for (int j = t; j <= k; j += kCoefThreads) coef[j] = 0.0;
            if (t == 0) {
                s[k] = sk;
                state[0] = (double)k;
            }
        }
    } else {
        // new row k of Linv: -(l^T Linv[0:k][0:k]) / lam, then 1 / lam; z_k = <row k, c>;
        // y = Linv^T z, coef_j = y_j s_j: each CTA a share of the columns
        const double ilam = rsqrt(fmax(gk - ll, 1e-300));
        const double zk = (ck - lz) * ilam;
        double *rowk = Linv + (int64_t)k * ldl;
        for (int j = rank * kCoefThreads + t; j < k; j += kCoefCtas * kCoefThreads) {
            double a = 0.0, b = 0.0;
#pragma unroll
            for (int r = 0; r < kCoefCtas; ++r) {
                const double *rg = cluster.map_shared_rank(g, r);
                a += rg[j];
                b += rg[k + 1 + j];
            }
            const double v = -a * ilam;
            rowk[j] = v;
            coef[j] = fma(zk, v, b) * s[j];
        }
        if (rank == 0) {
            if (off) atomicMax(reinterpret_cast<unsigned long long *>(state + 1), (unsigned long long)off);
            if (t == 0) {
                s[k] = sk;
                rowk[k] = ilam;
                coef[k] = zk * ilam * sk;
                alpha[k] = ck;
            }
        }
    }
    cluster.sync();        // no CTA leaves while its shared memory is read
}

}  // namespace ed

using namespace ed;

extern "C" int64_t ed_lanczos_state_doubles(int mmax)
{
    if (mmax < 1 || mmax > kLanczosMax) return -1;
    return lz_work_off(mmax) + 4 * (int64_t)(mmax + 1);
}

extern "C" int ed_lanczos_coef(void *stream, int k, int mmax, const double *dots, const double *nrm, double *state,
                               double *coef, double *alpha, double *beta)
{
    clear_error();
    ED_REQUIRE(mmax >= 1 && mmax <= kLanczosMax, "mmax=%d outside 1..%d", mmax, kLanczosMax);
    ED_REQUIRE(k >= 0 && k <= mmax, "step %d outside 0..%d", k, mmax);
    ED_REQUIRE(state != nullptr && alpha != nullptr && beta != nullptr, "state, alpha or beta is NULL");
    ED_REQUIRE(k == 0 || nrm != nullptr, "nrm is NULL");
    ED_REQUIRE(dots == nullptr || (coef != nullptr && k < mmax), "coef is NULL or step %d has no next vector", k);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return launch_coef(st, k, mmax, dots, 1, nrm, 1, state, coef, alpha, beta);
}

int ed::launch_coef(cudaStream_t st, int k, int mmax, const double *dots, int drows, const double *nrm, int nrows,
                    double *state, double *coef, double *alpha, double *beta)
{
    if (dots == nullptr) {
        lanczos_close_kernel<<<1, 32, 0, st>>>(k, nrm, state, alpha, beta);
        ED_CHECK_LAUNCH();
        return ED_OK;
    }
    const size_t smem = coef_smem(k);
    if (smem > 40 * 1024)      // the default limit of 48 KB holds the static arrays as well
        ED_CHECK_CUDA(cudaFuncSetAttribute(lanczos_coef_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)coef_smem(kLanczosMax)));
    lanczos_coef_kernel<<<kCoefCtas, kCoefThreads, smem, st>>>(k, mmax, dots, drows, nrm, nrows, state, coef,
                                                                alpha, beta);
    ED_CHECK_LAUNCH();
    return ED_OK;
}
