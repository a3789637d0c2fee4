// ed_vec.cu -- Krylov-space vector kernels: many dot products in one pass
// over the basis, and the projection update w - V c with its norm.
//
// These carry the Lanczos scalars of lanczos.f90:53-58 (DOT_PRODUCT, the
// three-term update, NORM2) and the full reorthogonalisation that the
// reference lacks (its LANCZOS_NORM, lanczos.f90:137-161, only measures the
// loss).  FP32 vectors: products are formed and summed in FP32 over 16
// elements per thread, every such partial is promoted to FP64 and all further
// accumulation is FP64, so no FP64 multiply is spent per element.  FP64
// vectors: FP64 throughout.  (The FP32 multi-dot reduces each warp's 512
// products in FP32 before the FP64 stage; see multidot32_kernel.)
#include "ed_common.cuh"

#include <algorithm>
#include <type_traits>

namespace ed {

int launch_reduce(const double *partials, int nblocks, int m, double *out, cudaStream_t st);

static constexpr int kVecThreads = 256;
static constexpr int kEPT = 16;                      // elements per thread per chunk
static constexpr int kChunk = kVecThreads * kEPT;    // 4096 elements
static constexpr int kMaxBlocks = 1024;
static_assert(kMaxNormRows <= 2 * kMaxBlocks, "the smallest scratch holds 2 * kMaxBlocks partial norms");
static constexpr int kVecResident = 4;               // CTAs per SM that a vector pass aims at

// Four consecutive elements p[i..i+3] (zeros past n); p is 16-byte aligned and i a multiple of 4.
template <typename T>
__device__ __forceinline__ void load4(T *r, const T *__restrict__ p, int64_t i, int64_t n)
{
    if (i + 3 < n) {
        if constexpr (sizeof(T) == 4) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(p + i));
            r[0] = v.x; r[1] = v.y; r[2] = v.z; r[3] = v.w;
        } else {
            const double2 v0 = __ldg(reinterpret_cast<const double2 *>(p + i));
            const double2 v1 = __ldg(reinterpret_cast<const double2 *>(p + i + 2));
            r[0] = v0.x; r[1] = v0.y; r[2] = v1.x; r[3] = v1.y;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) r[j] = (i + j < n) ? __ldg(p + i + j) : (T)0;
    }
}

// EPT elements of a thread: base + t*4 + k*4*NT + j (j < 4), k < EPT/4, in a CTA of NT threads.
template <typename T, int EPT, int NT>
__device__ __forceinline__ void load_chunk(T (&r)[EPT], const T *__restrict__ p, int64_t base, int64_t n)
{
#pragma unroll
    for (int k = 0; k < EPT / 4; ++k) load4<T>(r + 4 * k, p, base + (int64_t)k * (NT * 4) + threadIdx.x * 4, n);
}

// FP32: partials[block][j] (j < nvec) = sum over the block's chunks of <V_j, w>,
// partials[block][nvec + j] the same with z (when z != NULL).
// Each warp forms its 512 products per chunk and reduces them in
// FP32 (shuffles); only that warp partial is promoted and added in FP64, so
// the FP64 work is one add per 512 elements and vector.  For random-sign
// data the FP32 stage contributes an absolute error ~eps32 |V_j||w|/sqrt(n).
// Bound by HBM once the chunks fill the chip.  A vector shorter than that (fewer chunks than
// kVecResident CTAs per SM) splits the basis over blockIdx.y, jper vectors each, so that its pass
// is a few vectors deep instead of all of them (100 vectors of 63,488: 72 -> 19 us; of 853,872:
// 117 -> 74 us; 11.8 M and more: unchanged, 6.6-6.9 TB/s).
__global__ void __launch_bounds__(kVecThreads, kVecResident) multidot32_kernel(int64_t n, const float *__restrict__ V, int64_t ldv,
                                                                 int nvec, int jper, const float *__restrict__ w,
                                                                 const float *__restrict__ z,
                                                                 double *__restrict__ partials)
{
    extern __shared__ double acc[];  // [8 warps][mj]
    const int j0 = blockIdx.y * jper, nj = min(jper, nvec - j0);
    const int m = z ? 2 * nvec : nvec, mj = z ? 2 * nj : nj;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int j = threadIdx.x; j < 8 * mj; j += blockDim.x) acc[j] = 0.0;
    __syncthreads();
    const int64_t nchunks = (n + kChunk - 1) / kChunk;
    for (int64_t ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
        const int64_t base = ch * kChunk;
        float rw[kEPT], rz[kEPT];
        load_chunk<float, kEPT, kVecThreads>(rw, w, base, n);
        if (z) load_chunk<float, kEPT, kVecThreads>(rz, z, base, n);
#pragma unroll 2
        for (int j = 0; j < nj; ++j) {
            float rv[kEPT];
            load_chunk<float, kEPT, kVecThreads>(rv, V + (int64_t)(j0 + j) * ldv, base, n);
            float pw = 0, pz = 0;
#pragma unroll
            for (int k = 0; k < kEPT; ++k) pw += rv[k] * rw[k];
            if (z) {
#pragma unroll
                for (int k = 0; k < kEPT; ++k) pz += rv[k] * rz[k];
            }
            pw = warp_sumf(pw);
            if (z) pz = warp_sumf(pz);
            if (lane == 0) {
                acc[warp * mj + j] += (double)pw;
                if (z) acc[warp * mj + nj + j] += (double)pz;
            }
        }
    }
    __syncthreads();
    for (int j = threadIdx.x; j < mj; j += blockDim.x) {
        double s = 0.0;
        for (int q = 0; q < 8; ++q) s += acc[q * mj + j];
        partials[(int64_t)blockIdx.x * m + (j < nj ? j0 + j : nvec + j0 + j - nj)] = s;
    }
}

// FP64, same partials.  An FP64 instruction costs 64 FP32 ones on this chip, so the pass is bound by
// the FP64 pipe (two FMA per basis element) and spends it on nothing else: a CTA owns up to kJ64 vectors
// and one range of elements, every thread keeps its 2*kJ64 sums in registers over the whole range,
// and lanes are summed once at its end (the pass that summed lanes after every 16 elements took 11
// FP64 instructions per 8 here).  w and z are read again for every kJ64 vectors, from L2.
// NV = 0: groups of up to kJ64 vectors.  NV of 1 to 4: all nvec = NV vectors, where the loads are the time:
// U steps of all of them are in flight together (one vector of 1.7e8: 778 us as a group, 375 so; of
// 300,000: 9.5 -> 4.9).  One wave of CTAs has less to start and to sum than two (seven of 500,000 and z:
// 29.5 -> 23.6 us).
static constexpr int kJ64 = 8;
static constexpr int kStep64 = kVecThreads * 2;   // elements of one iteration: a 16-byte load per thread

__device__ __forceinline__ double2 load2(const double *__restrict__ p, int64_t i, int64_t n)
{
    if (i + 1 < n) return __ldg(reinterpret_cast<const double2 *>(p + i));
    return make_double2(i < n ? __ldg(p + i) : 0.0, 0.0);
}

// Sums of N values over the 32 lanes (N a power of two <= 32): each exchange halves the values a
// lane holds, so N sums cost about N additions instead of 5 N.  Value q ends in v[0] of lane
// q * (32 / N) (and its copies).
template <int N>
__device__ __forceinline__ void warp_sum_many(double (&v)[N])
{
    const int lane = threadIdx.x & 31;
    int o = 16;
#pragma unroll
    for (int h = N / 2; h >= 1; h >>= 1, o >>= 1) {
        const bool hi = (lane & o) != 0;
#pragma unroll
        for (int q = 0; q < N / 2; ++q) {
            if (q >= h) break;
            const double mine = hi ? v[q + h] : v[q], other = hi ? v[q] : v[q + h];
            v[q] = mine + __shfl_xor_sync(0xffffffffu, other, o);
        }
    }
    for (; o >= 1; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
}

// CTAs of a variant that an SM holds (registers)
template <int NV> constexpr int multidot64_ctas() { return NV == 1 ? 4 : NV ? 3 : 2; }

template <bool Z, int NV, int U>
__global__ void __launch_bounds__(kVecThreads, multidot64_ctas<NV>()) multidot64_kernel(int64_t n,
                                                                    const double *__restrict__ V, int64_t ldv, int nvec,
                                                                    const double *__restrict__ w,
                                                                    const double *__restrict__ z,
                                                                    double *__restrict__ partials)
{
    constexpr int M = NV ? NV : kJ64, KJ = M == 3 ? 4 : M;      // vectors, and their sums (a power of two)
    constexpr int NS = Z ? 2 * KJ : KJ;
    __shared__ double red[kVecThreads / 32][NS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ng = gridDim.y;
    const int j0 = NV ? 0 : (int)((int64_t)nvec * blockIdx.y / ng);
    const int nj = NV ? NV : (int)((int64_t)nvec * (blockIdx.y + 1) / ng) - j0;
    const int64_t steps = (n + U * kStep64 - 1) / (U * kStep64);
    const int64_t s0 = steps * blockIdx.x / gridDim.x, s1 = steps * (blockIdx.x + 1) / gridDim.x;
    double acc[NS];
#pragma unroll
    for (int q = 0; q < NS; ++q) acc[q] = 0.0;
    const double *Vj = V + (int64_t)j0 * ldv;
    for (int64_t st = s0; st < s1; ++st) {
        const int64_t i = st * (U * kStep64) + threadIdx.x * 2;
        double2 v[U][M], a[U], b[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int j = 0; j < M; ++j)
                if (j < nj) v[u][j] = load2(Vj + (int64_t)j * ldv, i + u * kStep64, n);
            a[u] = load2(w, i + u * kStep64, n);
            if constexpr (Z) b[u] = load2(z, i + u * kStep64, n);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int j = 0; j < M; ++j) {
                if (j >= nj) break;
                acc[j] = fma(v[u][j].x, a[u].x, acc[j]);
                if constexpr (Z) acc[KJ + j] = fma(v[u][j].x, b[u].x, acc[KJ + j]);
                acc[j] = fma(v[u][j].y, a[u].y, acc[j]);
                if constexpr (Z) acc[KJ + j] = fma(v[u][j].y, b[u].y, acc[KJ + j]);
            }
    }
    warp_sum_many<NS>(acc);
    if (lane % (32 / NS) == 0) red[warp][lane / (32 / NS)] = acc[0];
    __syncthreads();
    const int q = threadIdx.x, j = q % KJ;
    if (q < NS && j < nj) {
        double s = 0.0;
        for (int k = 0; k < kVecThreads / 32; ++k) s += red[k][q];
        partials[(int64_t)blockIdx.x * (Z ? 2 * nvec : nvec) + (q < KJ ? 0 : nvec) + j0 + j] = s;
    }
}

// out = ws w - sum_j coef_j V_j (w may be NULL; ws = wscale[0], a device
// scalar, or 1 when wscale is NULL), optional partial <out,out>.
// Accumulation type A: FP32 for an FP32 basis with FP32 output, FP64 otherwise.
// EPT elements per thread, NT threads: 16 x 256 streams long vectors at the HBM rate (FP64: the FP64
// pipe's), 4 x 128 spreads shorter ones evenly over the SMs (FP64, 50 vectors of 853,888: 120 ->
// 91 us; launch_update has the line between them).
template <typename T, typename O, typename A, int EPT, int NT>
__global__ void __launch_bounds__(NT) update_kernel(int64_t n, const T *__restrict__ V, int64_t ldv,
                                                             int nvec, const double *__restrict__ coef,
                                                             const double *__restrict__ wscale, const O *w, O *out,
                                                             double *__restrict__ partials)
{
    extern __shared__ double cs_raw[];
    A *cs = reinterpret_cast<A *>(cs_raw);
    for (int j = threadIdx.x; j < nvec; j += blockDim.x) cs[j] = (A)coef[j];
    const A ws = wscale ? (A)wscale[0] : (A)1;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double nrm = 0.0;
    constexpr int64_t chunk = (int64_t)NT * EPT;
    const int64_t nchunks = (n + chunk - 1) / chunk;
    for (int64_t ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
        const int64_t base = ch * chunk;
        A r[EPT];
        if (w) {
            O rw[EPT];
            load_chunk<O, EPT, NT>(rw, w, base, n);
#pragma unroll
            for (int k = 0; k < EPT; ++k) r[k] = ws * (A)rw[k];
        } else {
#pragma unroll
            for (int k = 0; k < EPT; ++k) r[k] = (A)0;
        }
        auto subtract = [&](int j) {
            T rv[EPT];
            load_chunk<T, EPT, NT>(rv, V + (int64_t)j * ldv, base, n);
            const A c = cs[j];
#pragma unroll
            for (int k = 0; k < EPT; ++k) r[k] -= c * (A)rv[k];
        };
        if constexpr (EPT == 4) {
#pragma unroll 4
            for (int j = 0; j < nvec; ++j) subtract(j);
        } else {
            for (int j = 0; j < nvec; ++j) subtract(j);
        }
        O ro[EPT];
#pragma unroll
        for (int k = 0; k < EPT; ++k) ro[k] = (O)r[k];
#pragma unroll
        for (int k = 0; k < EPT / 4; ++k) {
            const int64_t i = base + (int64_t)k * (NT * 4) + threadIdx.x * 4;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (i + j < n) out[i + j] = ro[4 * k + j];
        }
        if (partials) {
            if constexpr (sizeof(O) == 4) {
                float p = 0.f;
#pragma unroll
                for (int k = 0; k < EPT; ++k) p += ro[k] * ro[k];
                nrm += (double)p;
            } else {
#pragma unroll
                for (int k = 0; k < EPT; ++k) nrm += (double)ro[k] * (double)ro[k];
            }
        }
    }
    if (partials) {
        __shared__ double red[NT / 32];
        nrm = warp_sum(nrm);
        if (lane == 0) red[warp] = nrm;
        __syncthreads();
        if (threadIdx.x == 0) {
            double s = 0.0;
            for (int q = 0; q < NT / 32; ++q) s += red[q];
            partials[blockIdx.x] = s;
        }
    }
}

// The same for short vectors, where the chain of nvec loads is the time: a CTA's eight warps take
// every eighth vector of one 128-element tile each, and their sums meet in shared memory
// (FP64, 50 vectors of 4,928: 65 -> 14 us; of 63,488: 61 -> 18 us, most of it the two launches).
static constexpr int kSplitTile = 128;

template <typename T, typename O, typename A>
__global__ void __launch_bounds__(kVecThreads) update_split_kernel(int64_t n, const T *__restrict__ V, int64_t ldv,
                                                                   int nvec, const double *__restrict__ coef,
                                                                   const double *__restrict__ wscale, const O *w,
                                                                   O *out, double *__restrict__ partials)
{
    __shared__ __align__(16) A sums[8][kSplitTile];
    __shared__ double red[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const A ws = wscale ? (A)wscale[0] : (A)1;
    const int64_t ntiles = (n + kSplitTile - 1) / kSplitTile;
    double nrm = 0.0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t i = tile * kSplitTile + lane * 4;
        A r[4] = {0, 0, 0, 0};
#pragma unroll 4
        for (int j = warp; j < nvec; j += 8) {
            T rv[4];
            load4<T>(rv, V + (int64_t)j * ldv, i, n);
            const A c = (A)__ldg(coef + j);
#pragma unroll
            for (int k = 0; k < 4; ++k) r[k] += c * (A)rv[k];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) sums[warp][lane * 4 + k] = r[k];
        __syncthreads();
        const int64_t e = tile * kSplitTile + threadIdx.x;
        if (threadIdx.x < kSplitTile && e < n) {
            A s = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) s += sums[q][threadIdx.x];
            const O o = (O)((w ? ws * (A)w[e] : (A)0) - s);
            out[e] = o;
            nrm += (double)o * (double)o;
        }
        __syncthreads();
    }
    if (partials) {
        nrm = warp_sum(nrm);
        if (lane == 0) red[warp] = nrm;
        __syncthreads();
        if (threadIdx.x == 0) {
            double s = 0.0;
            for (int q = 0; q < 8; ++q) s += red[q];
            partials[blockIdx.x] = s;
        }
    }
}

static int64_t vec_ctas() { return std::min<int64_t>((int64_t)num_sms() * kVecResident, kMaxBlocks); }

// Partial rows of the multi-dot's grid (z or not) in *rows; the partials hold rows * m doubles.
int launch_multidot(cudaStream_t st, int dtype, int64_t n, const void *V, int64_t ldv, int nvec, const void *w,
                    const void *z, double *part, int *rows)
{
    const int64_t ctas = vec_ctas();
    if (dtype == ED_F32) {
        const int64_t nchunks = (n + kChunk - 1) / kChunk;
        const int gx = (int)std::max<int64_t>(1, std::min(nchunks, ctas));
        // one pass over all vectors once the chunks alone fill the chip (w and z are read once);
        // below that, groups of at least 4 vectors per CTA row
        int ng = (int)std::min<int64_t>((nvec + 3) / 4, std::max<int64_t>(1, ctas / gx));
        const int jper = (nvec + ng - 1) / ng;
        ng = (nvec + jper - 1) / jper;
        const size_t smem = sizeof(double) * 8 * (size_t)jper * (z ? 2 : 1);
        if (smem > 48 * 1024)
            ED_CHECK_CUDA(cudaFuncSetAttribute(multidot32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)smem));
        multidot32_kernel<<<dim3((unsigned)gx, (unsigned)ng), kVecThreads, smem, st>>>(
            n, static_cast<const float *>(V), ldv, nvec, jper, static_cast<const float *>(w),
            static_cast<const float *>(z), part);
        *rows = gx;
    } else {
        const double *Vd = static_cast<const double *>(V), *wd = static_cast<const double *>(w),
                     *zd = static_cast<const double *>(z);
        int ng = 1, gx = 0;
        // one group: a wave of resident CTAs; several groups, of unequal sizes: two.  One CTA more than
        // whole waves costs a wave
        auto launch = [&](auto count, auto un) {
            constexpr int NV = decltype(count)::value, U = decltype(un)::value;
            const int64_t steps = (n + U * kStep64 - 1) / (U * kStep64);
            const int64_t fill = ng == 1 ? (int64_t)num_sms() * multidot64_ctas<NV>() : ctas;
            gx = (int)std::max<int64_t>(1, std::min(steps, std::min(fill, ctas) / ng));
            const dim3 grid((unsigned)gx, (unsigned)ng);
            if (z) multidot64_kernel<true, NV, U><<<grid, kVecThreads, 0, st>>>(n, Vd, ldv, nvec, wd, zd, part);
            else multidot64_kernel<false, NV, U><<<grid, kVecThreads, 0, st>>>(n, Vd, ldv, nvec, wd, zd, part);
        };
        using std::integral_constant;
        // up to a step per SM there is nothing to keep in flight (4,928 elements, two vectors and z: 5.5 us, with
        // four steps 6.5)
        const int few = nvec <= 4 && n > (int64_t)kStep64 * num_sms() ? nvec : 0;
        if (few == 1) {
            launch(integral_constant<int, 1>(), integral_constant<int, 4>());
        } else if (few == 2) {
            launch(integral_constant<int, 2>(), integral_constant<int, 4>());
        } else if (few == 3) {
            launch(integral_constant<int, 3>(), integral_constant<int, 2>());
        } else if (few == 4) {
            launch(integral_constant<int, 4>(), integral_constant<int, 2>());
        } else {
            // groups of 5 to kJ64 vectors, as even as they come: the CTAs with the largest group end the pass
            ng = (nvec + kJ64 - 1) / kJ64;
            for (int g = ng + 1; g <= (nvec + 4) / 5; ++g)
                if ((int64_t)((nvec + g - 1) / g) * g < (int64_t)((nvec + ng - 1) / ng) * ng) ng = g;
            launch(integral_constant<int, 0>(), integral_constant<int, 1>());
        }
        *rows = gx;
    }
    ED_CHECK_LAUNCH();
    return ED_OK;
}

template <typename T, typename O, typename A>
static int launch_update(cudaStream_t st, int64_t n, const T *V, int64_t ldv, int nvec, const double *coef,
                         const double *wscale, const O *w, O *out, double *part, int *rows)
{
    const int64_t ctas = vec_ctas();
    const size_t smem = sizeof(double) * (size_t)(nvec > 0 ? nvec : 1);
    const int64_t tiles = (n + kSplitTile - 1) / kSplitTile;
    // The split form takes short vectors (up to four tiles per CTA) with vectors enough to pay for the exchange;
    // where its many partial norms have to be summed as well, that pays later.  Without a norm,
    // FP32: 63,488 elements, 7 vectors, 2.3 us against 3.3 for 4 x 128, 300,000 16 5.5 / 5.5; FP64: 20,000 2 2.7 /
    // 2.8, 63,488 8 4.5 / 4.6, 300,000 50 38.1 / 38.8.  With, FP32: 63,488 12 6.6 / 6.5, 300,000 50 14.7 / 15.5; FP64:
    // 63,488 24 10.8 / 11.4, 300,000 64 49 / 52; one vector of 300,000 8.7 / 6.0 and 14.1 / 7.3.
    // 4 x 128 takes the rest up to where 16-element chunks fill every resident CTA (FP64, bound by its pipe;
    // half of that for up to three vectors: one of 2.5 M 17 us, 16 x 256 14), or (FP32, bound by the streams)
    // while its chunks have a CTA each: 853,888 elements, 7 vectors, 4.2 / 5.1, 1.1 M 100 119 / 82.  With a
    // norm the fewer partial norms of 16 x 256 count: 853,888 12 11.1 / 9.6, 32 24.4 / 28.6.
    // (The steps of one Lanczos run take one form, whoever sums the norms: their vectors are the same.)
    const int64_t chunks = (n + kChunk - 1) / kChunk, ns = num_sms();
    constexpr bool f64 = sizeof(A) == 8;
    const bool norm = part != nullptr;
    int64_t split_from;
    if (norm) split_from = tiles <= 2 * ns ? 4 : f64 ? (tiles <= 4 * ns ? 24 : 64) : tiles / 45;
    else split_from = f64 ? (tiles <= 2 * ns ? 2 : tiles <= 4 * ns ? 8 : 48) : (tiles <= 4 * ns ? 1 : tiles / 150);
    const bool small = f64 ? chunks < (nvec > 3 ? ctas : ctas / 2)
                           : (n + 511) / 512 <= kMaxNormRows && (!norm || 9 * (int64_t)nvec >= chunks);
    if (tiles <= 4 * ctas && nvec >= split_from) {
        *rows = (int)std::min(tiles, ctas);
        update_split_kernel<T, O, A><<<*rows, kVecThreads, 0, st>>>(n, V, ldv, nvec, coef, wscale, w, out, part);
    } else if (small) {
        *rows = (int)std::min<int64_t>((n + 511) / 512, kMaxNormRows);
        update_kernel<T, O, A, 4, 128><<<*rows, 128, smem, st>>>(n, V, ldv, nvec, coef, wscale, w, out, part);
    } else {
        *rows = (int)std::min<int64_t>(chunks, ctas);
        update_kernel<T, O, A, kEPT, kVecThreads><<<*rows, kVecThreads, smem, st>>>(n, V, ldv, nvec, coef, wscale, w,
                                                                                    out, part);
    }
    ED_CHECK_LAUNCH();
    return ED_OK;
}

int launch_update_same(cudaStream_t st, int dtype, int64_t n, const void *V, int64_t ldv, int nvec, const double *coef,
                       const double *wscale, const void *w, void *out, double *part, int *rows)
{
    if (dtype == ED_F32)
        return launch_update<float, float, float>(st, n, static_cast<const float *>(V), ldv, nvec, coef, wscale,
                                                  static_cast<const float *>(w), static_cast<float *>(out), part, rows);
    return launch_update<double, double, double>(st, n, static_cast<const double *>(V), ldv, nvec, coef, wscale,
                                                 static_cast<const double *>(w), static_cast<double *>(out), part, rows);
}

}  // namespace ed

using namespace ed;

extern "C" int ed_multidot(void *stream, int dtype, int64_t n, const void *V, int64_t ldv, int nvec, const void *w,
                           const void *z, double *out, void *scratch, int64_t scratch_bytes)
{
    clear_error();
    ED_REQUIRE(dtype == ED_F32 || dtype == ED_F64, "dtype must be ED_F32 or ED_F64");
    ED_REQUIRE(n >= 0 && nvec >= 0, "negative size");
    ED_REQUIRE(out != nullptr, "out is NULL");
    if (nvec == 0 || n == 0) {
        if (nvec > 0) ED_CHECK_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * (z ? 2 : 1) * nvec, (cudaStream_t)stream));
        return ED_OK;
    }
    ED_REQUIRE(V != nullptr && w != nullptr, "V or w is NULL");
    ED_REQUIRE(ldv >= n, "ldv=%lld below n=%lld", (long long)ldv, (long long)n);
    const size_t esz = dtype == ED_F32 ? 4 : 8;
    ED_REQUIRE((reinterpret_cast<uintptr_t>(V) % 16) == 0 && (reinterpret_cast<uintptr_t>(w) % 16) == 0 &&
                   (!z || (reinterpret_cast<uintptr_t>(z) % 16) == 0) && ((ldv * esz) % 16) == 0,
               "V, w, z and the vector stride must be 16-byte aligned");
    ED_REQUIRE(scratch != nullptr && scratch_bytes >= ed_scratch_bytes(n, nvec),
               "scratch of %lld bytes is below the %lld needed", (long long)scratch_bytes,
               (long long)ed_scratch_bytes(n, nvec));
    const int m = z ? 2 * nvec : nvec;
    const size_t smem = sizeof(double) * 8 * (size_t)m;
    ED_REQUIRE(smem <= 200 * 1024, "nvec=%d too large for one pass", nvec);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double *part = static_cast<double *>(scratch);
    int rows = 0;
    const int rc = launch_multidot(st, dtype, n, V, ldv, nvec, w, z, part, &rows);
    if (rc) return rc;
    return launch_reduce(part, rows, m, out, st);
}

extern "C" int ed_update_wscaled(void *stream, int dtype, int out_dtype, int64_t n, const void *V, int64_t ldv,
                                 int nvec, const double *coef, const double *wscale, const void *w, void *out,
                                 double *norm2, void *scratch, int64_t scratch_bytes)
{
    clear_error();
    ED_REQUIRE(dtype == ED_F32 || dtype == ED_F64, "dtype must be ED_F32 or ED_F64");
    ED_REQUIRE(out_dtype == ED_F32 || out_dtype == ED_F64, "out_dtype must be ED_F32 or ED_F64");
    ED_REQUIRE(n >= 0 && nvec >= 0, "negative size");
    ED_REQUIRE(out != nullptr, "out is NULL");
    ED_REQUIRE(nvec == 0 || (V != nullptr && coef != nullptr), "V or coef is NULL");
    ED_REQUIRE(nvec == 0 || ldv >= n, "ldv=%lld below n=%lld", (long long)ldv, (long long)n);
    const size_t esz = dtype == ED_F32 ? 4 : 8, osz = out_dtype == ED_F32 ? 4 : 8;
    ED_REQUIRE((nvec == 0 || ((reinterpret_cast<uintptr_t>(V) % 16) == 0 && ((ldv * esz) % 16) == 0)) &&
                   (reinterpret_cast<uintptr_t>(out) % 16) == 0 && (!w || (reinterpret_cast<uintptr_t>(w) % 16) == 0),
               "V, w, out and the vector stride must be 16-byte aligned");
    (void)osz;
    ED_REQUIRE(nvec <= 8192, "nvec=%d too large", nvec);
    if (norm2) {
        ED_REQUIRE(scratch != nullptr && scratch_bytes >= ed_scratch_bytes(n, 1),
                   "scratch of %lld bytes is below the %lld needed", (long long)scratch_bytes,
                   (long long)ed_scratch_bytes(n, 1));
    }
    if (n == 0) return ED_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double *part = norm2 ? static_cast<double *>(scratch) : nullptr;
    int rows = 0, rc;
    if (dtype == ED_F32 && out_dtype == ED_F32)
        rc = launch_update<float, float, float>(st, n, static_cast<const float *>(V), ldv, nvec, coef, wscale,
                                                static_cast<const float *>(w), static_cast<float *>(out), part, &rows);
    else if (dtype == ED_F32 && out_dtype == ED_F64)
        rc = launch_update<float, double, double>(st, n, static_cast<const float *>(V), ldv, nvec, coef, wscale,
                                                  static_cast<const double *>(w), static_cast<double *>(out), part,
                                                  &rows);
    else if (dtype == ED_F64 && out_dtype == ED_F64)
        rc = launch_update<double, double, double>(st, n, static_cast<const double *>(V), ldv, nvec, coef, wscale,
                                                   static_cast<const double *>(w), static_cast<double *>(out), part,
                                                   &rows);
    else
        rc = launch_update<double, float, double>(st, n, static_cast<const double *>(V), ldv, nvec, coef, wscale,
                                                  static_cast<const float *>(w), static_cast<float *>(out), part,
                                                  &rows);
    if (rc) return rc;
    if (norm2) return launch_reduce(part, rows, 1, norm2, st);
    return ED_OK;
}

extern "C" int ed_update(void *stream, int dtype, int out_dtype, int64_t n, const void *V, int64_t ldv, int nvec,
                         const double *coef, const void *w, void *out, double *norm2, void *scratch,
                         int64_t scratch_bytes)
{
    return ed_update_wscaled(stream, dtype, out_dtype, n, V, ldv, nvec, coef, nullptr, w, out, norm2, scratch,
                             scratch_bytes);
}

// ---------------------------------------------------------------------------
// ed_multidot_noalloc: the multi-dot for callers that cannot allocate device
// memory and so cannot hand ed_multidot a scratch buffer.  Its per-block
// partial sums live in a fixed file-scope device array instead.

#include <mutex>

namespace ed {

constexpr int kNoAllocMaxNvec = 64;
constexpr int64_t kNoAllocDoubles = (int64_t)kMaxBlocks * 2 * kNoAllocMaxNvec;  // 131072 doubles = 1 MiB

// Partial sums of ed_multidot_noalloc.  Every GPU on which this library's
// kernels are loaded holds these 1 MiB until the process exits.  All calls on
// a device share the array: calls that overlap on the GPU race.  The kernel
// writes every partial before the reduction reads it, so nothing is cleared
// between calls.
static __device__ __align__(256) double g_noalloc_partials[kNoAllocDoubles];

constexpr int kNoAllocMaxDevices = 64;
static double *g_noalloc_addr[kNoAllocMaxDevices];
static std::mutex g_noalloc_mu;

// Device address of g_noalloc_partials on the current device.  In host code
// the array's name is only a host-side stand-in, so the address is looked up
// with the device current.  Outside a stream capture it is looked up on every
// call (cheap), so a context that was torn down and rebuilt, where the module
// may have loaded at another address, never gets a stale pointer; inside a
// capture the address cached by an earlier call on this device is used, and a
// capture with no earlier call is refused.
static int noalloc_partials(cudaStream_t st, double **out)
{
    int dev = 0;
    ED_CHECK_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices) {
        set_error("device %d is beyond the %d devices ed_multidot_noalloc tracks", dev, kNoAllocMaxDevices);
        return ED_ERR_RANGE;
    }
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    ED_CHECK_CUDA(cudaStreamIsCapturing(st, &cs));
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (cs == cudaStreamCaptureStatusNone) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_partials);
        if (e != cudaSuccess) {
            set_error("cudaGetSymbolAddress of the fixed scratch array failed: %s", cudaGetErrorString(e));
            return ED_ERR_CUDA;
        }
        g_noalloc_addr[dev] = static_cast<double *>(p);
    } else if (g_noalloc_addr[dev] == nullptr) {
        set_error("ed_multidot_noalloc: call it once on this device outside a stream capture first");
        return ED_ERR_ARG;
    }
    *out = g_noalloc_addr[dev];
    return ED_OK;
}

}  // namespace ed

extern "C" int ed_multidot_noalloc(void *stream, int dtype, int64_t n, const void *V, int64_t ldv, int nvec,
                                   const void *w, const void *z, double *out)
{
    clear_error();
    ED_REQUIRE(dtype == ED_F32 || dtype == ED_F64, "dtype must be ED_F32 or ED_F64");
    ED_REQUIRE(n >= 0 && nvec >= 0, "negative size");
    ED_REQUIRE(out != nullptr, "out is NULL");
    if (nvec > kNoAllocMaxNvec) {
        set_error("nvec=%d exceeds the %d vectors of ed_multidot_noalloc (its scratch is a fixed %lld-byte "
                  "device array); use ed_multidot with a scratch buffer for more",
                  nvec, kNoAllocMaxNvec, (long long)(kNoAllocDoubles * (int64_t)sizeof(double)));
        return ED_ERR_RANGE;
    }
    if (nvec == 0 || n == 0) {
        if (nvec > 0) ED_CHECK_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * (z ? 2 : 1) * nvec, (cudaStream_t)stream));
        return ED_OK;
    }
    ED_REQUIRE(V != nullptr && w != nullptr, "V or w is NULL");
    ED_REQUIRE(ldv >= n, "ldv=%lld below n=%lld", (long long)ldv, (long long)n);
    const size_t esz = dtype == ED_F32 ? 4 : 8;
    ED_REQUIRE((reinterpret_cast<uintptr_t>(V) % 16) == 0 && (reinterpret_cast<uintptr_t>(w) % 16) == 0 &&
                   (!z || (reinterpret_cast<uintptr_t>(z) % 16) == 0) && ((ldv * esz) % 16) == 0,
               "V, w, z and the vector stride must be 16-byte aligned");
    const int m = z ? 2 * nvec : nvec;
    // a grid has at most kMaxBlocks partial rows
    static_assert((int64_t)kMaxBlocks * 2 * kNoAllocMaxNvec <= kNoAllocDoubles, "partials exceed the fixed scratch");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double *part = nullptr;
    int rc = noalloc_partials(st, &part);
    if (rc) return rc;
    int rows = 0;
    rc = launch_multidot(st, dtype, n, V, ldv, nvec, w, z, part, &rows);
    if (rc) return rc;
    return launch_reduce(part, rows, m, out, st);
}
