// ed_hv.cu -- on-the-fly Hamiltonian-vector products.
//
// Hubbard (replaces HPROD, hprod_hubbard.f90:17-118).  With the vector viewed
// as a matrix X[d][u] (row = down string, contiguous up strings), H = A_up
// acting inside each row + A_dn mixing rows + a diagonal:
//   y[d][u] = diag(d,u) x[d][u] + sum_{q in up(u)} c x[d][q] + sum_{e in dn(d)} c x[e][u]
// Pass 1 (row pass): each CTA stages whole rows of x in shared memory and
//   applies the diagonal and the up hops from there (gathers stay on chip).
// Pass 2 (slab pass): the down hops are row-axpys y[d][:] += c x[e][:].
//   Columns are cut into slabs so that one slab of x (nsdn rows x slab
//   width) stays resident in L2 while every output row of that slab gathers
//   its ~N neighbour rows; x therefore streams from HBM about once.  The pass
//   also forms <x,y> and <y,y> for the Lanczos scalars.
//
// Heisenberg (replaces HPROD, hprod_heis.f90:1-61): ed_heis.cu, on the same
// row/pass structure (rows of B-half patterns over A-half patterns).
#include "ed_common.cuh"

#include <algorithm>
#include <atomic>
#include <cstdlib>

namespace ed {

struct HubArgs {
    int64_t nsup, nsdn, ld;
    const uint32_t *ustr; const int32_t *uptr; const int32_t *usrc; const void *ucf; const void *uediag;
    const uint32_t *dstr; const int32_t *dptr; const int32_t *dsrc; const void *dcf; const void *dediag;
    int64_t nslice;
    const int32_t *ell_off;        // of the type's table
    const int32_t *ell64_col, *ell64_src;
    const double *ell64_cf;
    const int2 *ell_pk32;          // or ell_sg32 (hop_slot)
    const int32_t *ell_sg32;
    float mag32[2];
    const void *u_lut;        // [4][256], then U times a count; float or double like the vectors
    int nbytes;               // bytes of a string with an on-site interaction (1 when there is none: zeros)
    int u_uniform, u_few;     // few: min(nup, ndn) < nbytes
    double u_value;
    double scale;
};

// on-site energy of the doubly occupied bits `both`, byte by byte from the table
template <typename T>
__device__ __forceinline__ T u_table(const HubArgs &a, uint32_t both)
{
    const T *lut = static_cast<const T *>(a.u_lut);
    T e = __ldg(lut + (both & 255u));
    for (int b = 1; b < a.nbytes; ++b) e += __ldg(lut + b * 256 + ((both >> (8 * b)) & 255u));
    return e;
}

// the same site by site
template <typename T>
__device__ __forceinline__ T u_by_site(const HubArgs &a, uint32_t both)
{
    const T *lut = static_cast<const T *>(a.u_lut);
    auto site = [&](int b) { return __ldg(lut + (b >> 3) * 256 + (1 << (b & 7))); };
    if (!both) return (T)0;
    T e = site(__ffs(both) - 1);
    for (both &= both - 1; both; both &= both - 1) e += site(__ffs(both) - 1);
    return e;
}

// the same; uval = U in T (uniform U, where a count is cheaper in FP32).  FEW: with fewer doubly occupied sites
// than bytes (u_few) a lane's sites cost the FP64 pipe less than the bytes (20 sites (2,6) 328 -> 294 us).
template <typename T, bool FEW = false>
__device__ __forceinline__ T u_energy(const HubArgs &a, uint32_t both, T uval)
{
    if (a.u_uniform) {
        if constexpr (sizeof(T) == 4) return uval * (T)__popc(both);
        return __ldg(static_cast<const T *>(a.u_lut) + 4 * 256 + __popc(both));   // no FP64 operation
    }
    if (FEW && a.u_few) return u_by_site<T>(a, both);
    return u_table<T>(a, both);
}

// Copy n elements from global src to shared dst (dst 16-byte aligned).
template <typename T>
__device__ __forceinline__ void stage_row(T *dst, const T *__restrict__ src, int64_t n, bool vec_ok)
{
    constexpr int VW = 16 / sizeof(T);
    using V = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
    if (vec_ok) {
        int64_t nv = (n + VW - 1) / VW;  // may read into the zero padding of the row
        const V *s4 = reinterpret_cast<const V *>(src);
        V *d4 = reinterpret_cast<V *>(dst);
        for (int64_t i = threadIdx.x; i < nv; i += blockDim.x) d4[i] = __ldg(s4 + i);
    } else {
        for (int64_t i = threadIdx.x; i < n; i += blockDim.x) dst[i] = __ldg(src + i);
    }
}

// G up-hop slots of one lane (table entries at, at+32, ...) applied to the R
// staged rows; the G table loads are issued before the first gather (FP32:
// one packed 8-byte {source, coefficient} load per slot).
template <typename T, int R, int G, bool TWO>
__device__ __forceinline__ void row_group(const HubArgs &a, int64_t at, const T *xs, int64_t sld, T (&acc)[R])
{
    int q[G];
    T c[G];
#pragma unroll
    for (int i = 0; i < G; ++i) {
        if (sizeof(T) == 4) {
            float w;
            hop_slot<TWO>(a.ell_pk32, a.ell_sg32, a.mag32[0], a.mag32[1], at + i * 32, q[i], w);
            c[i] = (T)w;
        } else {
            q[i] = __ldg(a.ell64_src + at + i * 32);
            c[i] = (T)__ldg(a.ell64_cf + at + i * 32);
        }
    }
#pragma unroll
    for (int i = 0; i < G; ++i)
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] += c[i] * xs[r * sld + q[i]];
}

// Pass 1: diagonal + up hops, R rows per CTA iteration.  Each warp owns one
// 32-string slice at a time and walks its sliced-ELL slots (coalesced,
// four slots in flight), gathering the sources from the staged rows.
template <typename T, int R, bool TWO>
__global__ void __launch_bounds__(512, 2) hub_row_kernel(const T *__restrict__ x, T *__restrict__ y,
                                                      const HubArgs a, int64_t sld, int vec_ok)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *xs = reinterpret_cast<T *>(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int64_t nsup = a.nsup, ld = a.ld;
    const T uval = (T)a.u_value, sc = (T)a.scale;
    const T *ued_t = static_cast<const T *>(a.uediag), *ded_t = static_cast<const T *>(a.dediag);
    if (sizeof(T) == 4 && threadIdx.x < kZeroCols) {
#pragma unroll
        for (int r = 0; r < R; ++r) xs[r * sld + zero_col(nsup) + threadIdx.x] = (T)0;
    }
    for (int64_t d0 = (int64_t)blockIdx.x * R; d0 < a.nsdn; d0 += (int64_t)gridDim.x * R) {
        const int nr = (int)min((int64_t)R, a.nsdn - d0);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (r < nr) stage_row<T>(xs + r * sld, x + (d0 + r) * ld, nsup, vec_ok != 0);
        __syncthreads();
        uint32_t sd[R];
        T ed[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            sd[r] = (r < nr) ? __ldg(a.dstr + d0 + r) : 0u;
            ed[r] = (r < nr) ? __ldg(ded_t + d0 + r) : (T)0;
        }
        for (int64_t sl = warp; sl < a.nslice; sl += nwarps) {
            const int64_t u = sizeof(T) == 4 ? sl * 32 + lane : (int64_t)__ldg(a.ell64_col + sl * 32 + lane);
            const bool ok = sizeof(T) == 4 ? u < nsup : u >= 0;
            const int64_t uu = ok ? u : nsup - 1;
            const uint32_t su = __ldg(a.ustr + uu);
            const T eu = __ldg(ued_t + uu);
            T acc[R];
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = (eu + ed[r] + u_energy<T, sizeof(T) == 8>(a, su & sd[r], uval)) * xs[r * sld + uu];
            const int s0 = __ldg(a.ell_off + sl), ns = __ldg(a.ell_off + sl + 1) - s0;
            const int64_t at0 = (int64_t)s0 * 32 + lane;
            // slots in groups: all table loads of a group are in flight before its first gather
            int k = 0;
            for (; k + 8 <= ns; k += 8) row_group<T, R, 8, TWO>(a, at0 + k * 32, xs, sld, acc);
            if (k + 4 <= ns) {
                row_group<T, R, 4, TWO>(a, at0 + k * 32, xs, sld, acc);
                k += 4;
            }
            for (; k < ns; ++k) row_group<T, R, 1, TWO>(a, at0 + k * 32, xs, sld, acc);
            if (ok) {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (r < nr) y[(d0 + r) * ld + u] = (sc == (T)1) ? acc[r] : acc[r] * sc;
            }
        }
        __syncthreads();
    }
}

// Pass 1 for FP32 with four rows per CTA, column layout: the four rows of
// string u are staged as one 16-byte column xs4[u], so a hop gathers all four
// rows with one 128-bit shared load.  A quarter warp's 8 lanes hit 8 bank
// groups when their sources differ mod 8, which the sliced-ELL slot order
// arranges (ed_sector.cu, ell_order).
template <int G, bool TWO>
__device__ __forceinline__ void col_group(const HubArgs &a, int64_t at, const float4 *xs4, float (&acc)[4])
{
    int q[G];
    float c[G];
#pragma unroll
    for (int i = 0; i < G; ++i) {
        hop_slot<TWO>(a.ell_pk32, a.ell_sg32, a.mag32[0], a.mag32[1], at + i * 32, q[i], c[i]);
    }
#pragma unroll
    for (int i = 0; i < G; ++i) {
        const float4 v = xs4[q[i]];
        acc[0] += c[i] * v.x;
        acc[1] += c[i] * v.y;
        acc[2] += c[i] * v.z;
        acc[3] += c[i] * v.w;
    }
}

template <bool TWO>
__global__ void __launch_bounds__(1024) hub_row_col4_kernel(const float *__restrict__ x, float *__restrict__ y,
                                                            const HubArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float4 *xs4 = reinterpret_cast<float4 *>(smem_raw);   // [nsup], then the zero columns
    if (threadIdx.x < kZeroCols) xs4[zero_col(a.nsup) + threadIdx.x] = make_float4(0.f, 0.f, 0.f, 0.f);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int64_t nsup = a.nsup, ld = a.ld;
    const float uval = (float)a.u_value, sc = (float)a.scale;
    const float *ued_t = static_cast<const float *>(a.uediag), *ded_t = static_cast<const float *>(a.dediag);
    for (int64_t d0 = (int64_t)blockIdx.x * 4; d0 < a.nsdn; d0 += (int64_t)gridDim.x * 4) {
        const int nr = (int)min((int64_t)4, a.nsdn - d0);
        const float *x0 = x + d0 * ld;
        for (int64_t c = threadIdx.x; c < nsup; c += blockDim.x) {
            float4 v;
            v.x = __ldg(x0 + c);
            v.y = nr > 1 ? __ldg(x0 + ld + c) : 0.f;
            v.z = nr > 2 ? __ldg(x0 + 2 * ld + c) : 0.f;
            v.w = nr > 3 ? __ldg(x0 + 3 * ld + c) : 0.f;
            xs4[c] = v;
        }
        __syncthreads();
        uint32_t sd[4];
        float ed[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            sd[r] = (r < nr) ? __ldg(a.dstr + d0 + r) : 0u;
            ed[r] = (r < nr) ? __ldg(ded_t + d0 + r) : 0.f;
        }
        for (int64_t sl = warp; sl < a.nslice; sl += nwarps) {
            const int64_t u = sl * 32 + lane;
            const bool ok = u < nsup;
            const int64_t uu = ok ? u : nsup - 1;
            const uint32_t su = __ldg(a.ustr + uu);
            const float eu = __ldg(ued_t + uu);
            const float4 xv = xs4[uu];
            const float xr[4] = {xv.x, xv.y, xv.z, xv.w};
            float acc[4];
            if (a.u_uniform) {
#pragma unroll
                for (int r = 0; r < 4; ++r) acc[r] = (eu + ed[r] + uval * (float)__popc(su & sd[r])) * xr[r];
            } else {
#pragma unroll
                for (int r = 0; r < 4; ++r) acc[r] = (eu + ed[r] + u_table<float>(a, su & sd[r])) * xr[r];
            }
            const int s0 = __ldg(a.ell_off + sl), ns = __ldg(a.ell_off + sl + 1) - s0;
            const int64_t at0 = (int64_t)s0 * 32 + lane;
            int k = 0;
            for (; k + 8 <= ns; k += 8) col_group<8, TWO>(a, at0 + k * 32, xs4, acc);
            if (k + 4 <= ns) {
                col_group<4, TWO>(a, at0 + k * 32, xs4, acc);
                k += 4;
            }
            for (; k < ns; ++k) col_group<1, TWO>(a, at0 + k * 32, xs4, acc);
            if (ok) {
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (r < nr) y[(d0 + r) * ld + u] = acc[r] * sc;
            }
        }
        __syncthreads();
    }
}

// A down hop of a row: source row and coefficient.
template <typename T> struct alignas(sizeof(T) == 4 ? 8 : 16) RowHop {
    int src;
    T cf;
};

// Pass 2: down hops, y[d][slab] += sum_e c_e x[src_e][slab]; optional dots.
// Work items (slab, group of 8 rows) are visited slab-major by a persistent
// grid so that the CTAs in flight share one or two slabs of x in L2.  A warp
// keeps its row's neighbour list in shared memory (one 8- or 16-byte broadcast
// read per hop; two or three shuffles per hop before), walks U chunks of 32*VW columns together
// and issues the loads of L neighbour rows back to back.
template <typename T, int VW, int U, int L, bool SINGLE>
__global__ void __launch_bounds__(256) hub_slab_kernel(const T *__restrict__ x, T *__restrict__ y,
                                                       const HubArgs a, int slab_w, int ngroups, int nitems,
                                                       double *__restrict__ partials)
{
    __shared__ RowHop<T> lists[8][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    RowHop<T> *hop = lists[warp];
    const T *__restrict__ cf = static_cast<const T *>(a.dcf);
    const int nsup = (int)a.nsup;
    const int64_t ld = a.ld;
    const T sc = (T)a.scale;
    double dxy = 0.0, dyy = 0.0;
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const int slab = item / ngroups, d = (item - slab * ngroups) * 8 + warp;
        if (d >= a.nsdn) continue;
        const int c0 = slab * slab_w, c1 = min(c0 + slab_w, nsup);
        const int e0 = __ldg(a.dptr + d), nn = __ldg(a.dptr + d + 1) - e0;
        T *yr = y + (int64_t)d * ld;
        const T *xd = x + (int64_t)d * ld;
        float pxy = 0.f, pyy = 0.f;
        double qxy = 0.0, qyy = 0.0;
        auto dot = [&](T xv, T yv) {
            if constexpr (sizeof(T) == 4) { pxy += xv * yv; pyy += yv * yv; }
            else { qxy += xv * yv; qyy += yv * yv; }
        };
        for (int b0 = 0; b0 < nn; b0 += 32) {
            const int nb = min(32, nn - b0);
            __syncwarp();
            if (lane < nb) {
                hop[lane].src = __ldg(a.dsrc + e0 + b0 + lane);
                hop[lane].cf = __ldg(cf + e0 + b0 + lane) * sc;
            }
            __syncwarp();
            const bool last = (b0 + 32 >= nn);
            // UN chunks of 32*VW columns from cb on, NL neighbour rows' loads in flight
            auto pass = [&](auto chunks, auto loads, int cb) {
                constexpr int UN = decltype(chunks)::value, NL = decltype(loads)::value;
                using V = typename std::conditional<VW == 1, T, typename std::conditional<sizeof(T) == 4, float4, double2>::type>::type;
                const V *xc = reinterpret_cast<const V *>(x + cb) + lane;
                V *yc = reinterpret_cast<V *>(yr + cb) + lane;
                V acc[UN];
#pragma unroll
                for (int u = 0; u < UN; ++u) acc[u] = yc[u * 32];
                auto hops = [&](auto count, int e) {
                    constexpr int N = decltype(count)::value;
                    V v[N][UN];
                    T w[N];
#pragma unroll
                    for (int i = 0; i < N; ++i) {
                        const RowHop<T> h = hop[e + i];
                        w[i] = h.cf;
                        const V *xr = reinterpret_cast<const V *>(reinterpret_cast<const T *>(xc) + h.src * ld);
#pragma unroll
                        for (int u = 0; u < UN; ++u) v[i][u] = __ldg(xr + u * 32);
                    }
#pragma unroll
                    for (int i = 0; i < N; ++i)
#pragma unroll
                        for (int u = 0; u < UN; ++u)
#pragma unroll
                            for (int k = 0; k < VW; ++k)
                                reinterpret_cast<T *>(&acc[u])[k] += w[i] * reinterpret_cast<const T *>(&v[i][u])[k];
                };
                int e = 0;
                for (; e + NL <= nb; e += NL) hops(std::integral_constant<int, NL>(), e);
                if (NL > 2 && e + 2 <= nb) {
                    hops(std::integral_constant<int, 2>(), e);
                    e += 2;
                }
                for (; e < nb; ++e) hops(std::integral_constant<int, 1>(), e);
#pragma unroll
                for (int u = 0; u < UN; ++u) yc[u * 32] = acc[u];
                if (partials && last) {
#pragma unroll
                    for (int u = 0; u < UN; ++u) {
                        const V xv = __ldg(reinterpret_cast<const V *>(xd + cb) + lane + u * 32);
#pragma unroll
                        for (int k = 0; k < VW; ++k)
                            dot(reinterpret_cast<const T *>(&xv)[k], reinterpret_cast<const T *>(&acc[u])[k]);
                    }
                }
            };
            using std::integral_constant;
            int cb = c0;
            // whole passes of U chunks
            for (; cb + 32 * VW * U <= c1; cb += 32 * VW * U) pass(integral_constant<int, U>(), integral_constant<int, L>(), cb);
            if constexpr (SINGLE) {
                // whole chunks, then a short one of lanes with VW columns (not for 32 columns or fewer in FP64, where an
                // idle lane costs the pipe what a busy one does)
                constexpr int kAlone = sizeof(T) == 4 ? 0 : 32;
                for (; cb + 32 * VW <= c1; cb += 32 * VW) pass(integral_constant<int, 1>(), integral_constant<int, 4>(), cb);
                if (c1 - cb > kAlone) {
                    if (cb + (lane + 1) * VW <= c1) pass(integral_constant<int, 1>(), integral_constant<int, 4>(), cb);
                    cb += (c1 - cb) / VW * VW;
                }
            }
            // the rest of the slab, a column per lane
            for (int c = cb + lane; c < c1; c += 32) {
                T acc = yr[c];
#pragma unroll 4
                for (int e = 0; e < nb; ++e) acc += hop[e].cf * __ldg(x + hop[e].src * ld + c);
                yr[c] = acc;
                if (partials && last) dot(__ldg(xd + c), acc);
            }
        }
        if (nn == 0 && partials) {
            // no down hops: the dots still need this row's y
            for (int cc = c0 + lane; cc < c1; cc += 32) {
                dot(__ldg(xd + cc), yr[cc]);
            }
        }
        dxy += (double)pxy + qxy;
        dyy += (double)pyy + qyy;
    }
    if (partials) {
        __shared__ double red[2][8];
        dxy = warp_sum(dxy);
        dyy = warp_sum(dyy);
        if (lane == 0) { red[0][warp] = dxy; red[1][warp] = dyy; }
        __syncthreads();
        if (threadIdx.x == 0) {
            double sxy = 0.0, syy = 0.0;
            for (int w = 0; w < 8; ++w) { sxy += red[0][w]; syy += red[1][w]; }
            partials[2 * blockIdx.x] = sxy;
            partials[2 * blockIdx.x + 1] = syy;
        }
    }
}

// Both passes in one, for small sectors: R rows are staged side by side in shared memory, a thread owns
// one of them (its row constants stay in registers) and every blockDim/R-th column: diagonal, down
// hops from the neighbour rows in L2, up hops from the staged rows, scale, store, dots.  Bound by
// latency (a thread's loads for one column are in flight together, nothing else), which a launch less
// and no second trip of y outweigh while the sector is small.  Items (row block, column share) are cut
// so that every resident CTA walks several.  With ADD the product is added to y.
template <typename T, int R, bool ADD>
__global__ void __launch_bounds__(512, 2) hub_fused_kernel(const T *__restrict__ x, T *y, const HubArgs a, int maxrow,
                                                           int csplit, int64_t nitems, double *__restrict__ partials)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RowHop<T> *nb = reinterpret_cast<RowHop<T> *>(smem_raw);   // [R][maxrow]
    T *xs = reinterpret_cast<T *>(nb + R * maxrow);             // [nsup][R]
    const int nsup = (int)a.nsup;
    const int64_t ld = a.ld;
    const T sc = (T)a.scale;
    const T *ued_t = static_cast<const T *>(a.uediag), *ded_t = static_cast<const T *>(a.dediag);
    const T *ucf = static_cast<const T *>(a.ucf), *dcf = static_cast<const T *>(a.dcf);
    const int r = threadIdx.x % R, step = blockDim.x / R;
    double dxy = 0.0, dyy = 0.0;
    int64_t staged = -1;
    for (int64_t item = blockIdx.x; item < nitems; item += gridDim.x) {
        const int64_t rb = item / csplit;
        const int cs = (int)(item - rb * csplit);
        const int64_t d0 = rb * R, d = d0 + r;
        const bool row = d < a.nsdn;
        int nn = 0;
        if (row) nn = __ldg(a.dptr + d + 1) - __ldg(a.dptr + d);
        if (rb != staged) {
            __syncthreads();      // the previous rows' readers are done
            for (int i = threadIdx.x; i < nsup; i += blockDim.x) {
#pragma unroll
                for (int q = 0; q < R; ++q) xs[i * R + q] = (d0 + q < a.nsdn) ? __ldg(x + (d0 + q) * ld + i) : (T)0;
            }
            if (row) {
                const int e0 = __ldg(a.dptr + d);
                for (int e = threadIdx.x / R; e < nn; e += step) {
                    nb[r * maxrow + e].src = __ldg(a.dsrc + e0 + e);
                    nb[r * maxrow + e].cf = __ldg(dcf + e0 + e);
                }
            }
            staged = rb;
            __syncthreads();
        }
        if (!row) continue;
        const uint32_t sd = __ldg(a.dstr + d);
        const T ed = __ldg(ded_t + d);
        const RowHop<T> *hop = nb + r * maxrow;
        const int c0 = (int)((int64_t)nsup * cs / csplit), c1 = (int)((int64_t)nsup * (cs + 1) / csplit);
        T pxy = 0, pyy = 0;
        for (int c = c0 + threadIdx.x / R; c < c1; c += step) {
            const T xv = xs[c * R + r];
            T acc = (__ldg(ued_t + c) + ed + u_energy<T>(a, __ldg(a.ustr + c) & sd, (T)a.u_value)) * xv;
            const T *xc = x + c;
            int e = 0;
            for (; e + 4 <= nn; e += 4) {
                T v[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = __ldg(xc + hop[e + i].src * ld);
#pragma unroll
                for (int i = 0; i < 4; ++i) acc += hop[e + i].cf * v[i];
            }
            for (; e < nn; ++e) acc += hop[e].cf * __ldg(xc + hop[e].src * ld);
            const int u1 = __ldg(a.uptr + c + 1);
#pragma unroll 4
            for (int q = __ldg(a.uptr + c); q < u1; ++q) acc += __ldg(ucf + q) * xs[__ldg(a.usrc + q) * R + r];
            if (sc != (T)1) acc *= sc;
            T *yp = y + d * ld + c;
            if (ADD) acc += *yp;
            *yp = acc;
            if (partials) {
                pxy += xv * acc;
                pyy += acc * acc;
            }
        }
        dxy += (double)pxy;
        dyy += (double)pyy;
    }
    if (partials) {
        __shared__ double red[2][16];
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        dxy = warp_sum(dxy);
        dyy = warp_sum(dyy);
        if (lane == 0) { red[0][warp] = dxy; red[1][warp] = dyy; }
        __syncthreads();
        if (threadIdx.x == 0) {
            double sxy = 0.0, syy = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { sxy += red[0][w]; syy += red[1][w]; }
            partials[2 * blockIdx.x] = sxy;
            partials[2 * blockIdx.x + 1] = syy;
        }
    }
}

// Sum nblocks rows of m partials into out[m] (FP64, fixed order).
__global__ void reduce_partials_kernel(const double *__restrict__ partials, int nblocks, int m,
                                       double *__restrict__ out)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nw = blockDim.x >> 5;
    for (int j = blockIdx.x * nw + warp; j < m; j += gridDim.x * nw) {
        double s = 0.0;
        for (int b = lane; b < nblocks; b += 32) s += partials[(int64_t)b * m + j];
        s = warp_sum(s);
        if (lane == 0) out[j] = s;
    }
}

// The same for a few outputs of many rows: a CTA per output.
__global__ void __launch_bounds__(256) reduce_rows_kernel(const double *__restrict__ partials, int nblocks, int m,
                                                          double *__restrict__ out)
{
    __shared__ double red[8];
    const double s = sum_rows_cta(partials + blockIdx.x, nblocks, m, red);
    if (threadIdx.x == 0) out[blockIdx.x] = s;
}

int launch_reduce(const double *partials, int nblocks, int m, double *out, cudaStream_t st)
{
    if (m <= 8 && nblocks > 64) {
        reduce_rows_kernel<<<m, 256, 0, st>>>(partials, nblocks, m, out);
        ED_CHECK_LAUNCH();
        return ED_OK;
    }
    int threads = 256, per = threads / 32;
    int blocks = (m + per - 1) / per;
    if (blocks > 1024) blocks = 1024;
    reduce_partials_kernel<<<blocks, threads, 0, st>>>(partials, nblocks, m, out);
    ED_CHECK_LAUNCH();
    return ED_OK;
}

// The Heisenberg product lives in ed_heis.cu.

// ------------------------------------------------------------ launchers

static constexpr int kMaxPartialBlocks = 1024;

// Sectors that take the one-pass product.  Measured one pass / two: 8-site ring FP64 9.4 / 12.8 us (one launch
// instead of two), 11 sites half filled (213,444) FP64 22.5 / 26.7, FP32 11.9 / 18.5; 16 sites (3,3)
// (313,600) 28.7 / 26.7 and 16.4 / 13.9, 3x4 half filled 101 / 81 and 48 / 23.  Rows of at most 112
// strings leave most of a row CTA idle: 15 sites (2,7), 675,675 states, 38.7 / 45.7 and 22.3 / 27.4; 20 sites
// (1,8) 149 / 573 and 89 / 302.  Between that and 128 strings only FP32: 16 sites (2,5), 524,160 states, with
// per-site U 30.6 / 27.5 and 16.2 / 20.2, without 29.2 / 26.3 and 15.5 / 15.8; (2,8), 1.5 M states, 82 / 67 and 45 / 36.
constexpr int64_t kFuseStates = 1 << 18;
constexpr int64_t kFuseRow = 112, kFuseRowSmall = 128, kFuseRowStates = 1 << 20;

// L2 budget of one x slab in the slab pass.  The part of L2 near an SM holds it only while it is small:
// 4x4 FP32 (256 / 512 / 768 columns: 13 / 26 / 40 MB) 1,486 / 1,696 / 1,812 us the whole product, 16 sites
// (7,7) 12 / 23 / 47 MB 1,170 / 1,198 / 1,418 us.  FP64 is bound by its pipe: at budgets of 20 and 48 MB 14 sites
// and 4x4 are level, 15 sites (7,7) 2,485 and 2,538 us, 16 sites (7,7) 9,271 and 9,170.  The environment variable
// PYHUB_ED_SLAB_L2_BYTES overrides it for tuning.
static double slab_l2_bytes()
{
    static double v = []() {
        const char *e = std::getenv("PYHUB_ED_SLAB_L2_BYTES");
        const double d = e ? std::atof(e) : 0.0;
        return (d >= 1.0e6 && d <= 1.0e9) ? d : 20.0e6;
    }();
    return v;
}

// Largest shared memory a kernel may ask for on the current device.
int max_smem()
{
    static std::atomic<int> known[64];
    int dev = 0;
    cudaGetDevice(&dev);
    int v = (dev >= 0 && dev < 64) ? known[dev].load(std::memory_order_relaxed) : 0;
    if (v == 0) {
        cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (dev >= 0 && dev < 64) known[dev].store(v, std::memory_order_relaxed);
    }
    return v;
}

template <typename T, int R>
static int launch_fused(ed_sector *s, cudaStream_t st, const T *x, T *y, HubArgs &a, bool add, double *dots,
                        double *partials)
{
    const int nsm = num_sms(), maxrow = std::max(s->dn.max_row, 1);
    const size_t smem = (size_t)R * maxrow * sizeof(RowHop<T>) + (size_t)R * s->nsup * sizeof(T);
    auto *kfn = add ? hub_fused_kernel<T, R, true> : hub_fused_kernel<T, R, false>;
    if (smem > 48 * 1024)
        ED_CHECK_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // a thread a column (two to a thread keep two chains of loads in turn: 10 sites FP64 12.3 against 10.2 us)
    const int threads = (int)std::min<int64_t>(512, std::max<int64_t>(64, (R * s->nsup + 31) / 32 * 32));
    // CTAs resident per SM: by threads (at most 1024 by registers) and by shared memory
    const int per_sm = (int)std::max<int64_t>(1, std::min<int64_t>(1024 / threads, (228 * 1024) / (int64_t)(smem + 1024)));
    const int64_t rb = (s->nsdn + R - 1) / R, resident = std::min<int64_t>((int64_t)nsm * per_sm, kMaxPartialBlocks);
    const int64_t most = std::max<int64_t>(1, s->nsup * R / threads);    // a column for every thread
    const int csplit = (int)std::min<int64_t>(most, std::max<int64_t>(1, 6 * resident / rb));
    const int64_t nitems = rb * csplit, blocks = std::min(nitems, resident);
    kfn<<<(unsigned)blocks, threads, smem, st>>>(x, y, a, maxrow, csplit, nitems, dots ? partials : nullptr);
    ED_CHECK_LAUNCH();
    if (dots) return launch_reduce(partials, (int)blocks, 2, dots, st);
    return ED_OK;
}

// Bytes of a row's down hops in the one-pass kernel, and whether the sector takes it.
template <typename T> static size_t list_bytes(const ed_sector *s)
{
    return (size_t)std::max(s->dn.max_row, 1) * sizeof(RowHop<T>);
}

template <typename T> static bool one_pass(const ed_sector *s)
{
    const bool small = s->dim <= kFuseStates || s->nsup <= kFuseRow ||
                       (sizeof(T) == 4 && s->nsup <= kFuseRowSmall && s->dim <= kFuseRowStates);
    return small && list_bytes<T>(s) + (size_t)s->nsup * sizeof(T) <= (size_t)max_smem();
}

template <typename T>
static int hub_hv(ed_sector *s, cudaStream_t st, int64_t ld, const T *x, T *y, double scale, double *dots,
                  double *partials)
{
    HubArgs a;
    a.nsup = s->nsup; a.nsdn = s->nsdn; a.ld = ld;
    a.ustr = s->up.str; a.uptr = s->up.ptr; a.usrc = s->up.src;
    a.dstr = s->dn.str; a.dptr = s->dn.ptr; a.dsrc = s->dn.src;
    a.uediag = (sizeof(T) == 4) ? (const void *)s->up.ediag32 : (const void *)s->up.ediag;
    a.dediag = (sizeof(T) == 4) ? (const void *)s->dn.ediag32 : (const void *)s->dn.ediag;
    a.dcf = (sizeof(T) == 4) ? (const void *)s->dn.cf32 : (const void *)s->dn.cf64;
    a.ucf = (sizeof(T) == 4) ? (const void *)s->up.cf32 : (const void *)s->up.cf64;
    a.nslice = s->up.nslice;
    a.ell_off = (sizeof(T) == 4) ? s->up.ell_off : s->up.ell64_off;
    a.ell64_col = s->up.ell64_col;
    a.ell64_src = s->up.ell64_src;
    a.ell64_cf = s->up.ell64_cf;
    a.ell_pk32 = s->up.ell_pk32;
    a.ell_sg32 = s->up.ell_sg32;
    a.mag32[0] = s->up.mag32[0];
    a.mag32[1] = s->up.mag32[1];
    a.u_lut = (sizeof(T) == 4) ? (const void *)s->u_lut32 : (const void *)s->u_lut;
    a.nbytes = (s->u_uniform && s->u_value == 0.0) ? 1 : (s->norb + 7) / 8;
    a.u_uniform = s->u_uniform ? 1 : 0;
    a.u_few = std::min(s->nup, s->ndn) < a.nbytes ? 1 : 0;
    a.u_value = s->u_value;
    a.scale = scale;
    const int nsm = num_sms();
    constexpr int VWS = 16 / sizeof(T);
    // ---- pass 1
    const int64_t sld = sizeof(T) == 4 ? zero_col(s->nsup) + kZeroCols : (s->nsup + VWS - 1) / VWS * VWS;
    const bool vec_ok = (ld % VWS == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0);
    const int maxsm = max_smem();
    const size_t row_bytes = (size_t)sld * sizeof(T);
    if (row_bytes > (size_t)maxsm) {
        set_error("up-string row of %lld entries does not fit in shared memory (%d bytes)",
                  (long long)s->nsup, maxsm);
        return ED_ERR_RANGE;
    }
    const size_t lists = list_bytes<T>(s);
    if (one_pass<T>(s)) {
        // the U_ijkl terms go into a cleared y first, so that the dots see the whole product
        const bool add = s->uijkl != nullptr;
        if (add) {
            ED_CHECK_CUDA(cudaMemset2DAsync(y, (size_t)ld * sizeof(T), 0, (size_t)s->nsup * sizeof(T), (size_t)s->nsdn, st));
            const int rc = uijkl_hv(s, st, sizeof(T) == 4 ? ED_F32 : ED_F64, ld, x, y, scale);
            if (rc != ED_OK) return rc;
        }
        // four rows side by side, else two, where two CTAs of them fit an SM and the SMs have rows enough
        auto fits = [&](int R) {
            return R * (lists + s->nsup * sizeof(T)) <= (size_t)maxsm / 2 && s->nsdn >= (int64_t)R * nsm;
        };
        if (fits(4)) return launch_fused<T, 4>(s, st, x, y, a, add, dots, partials);
        if (fits(2)) return launch_fused<T, 2>(s, st, x, y, a, add, dots, partials);
        return launch_fused<T, 1>(s, st, x, y, a, add, dots, partials);
    }
    // FP32: four rows per 1024-thread CTA (one CTA per SM) when they fit, so every
    // hop-table slot serves four rows and one 128-bit gather reads all four;
    // else two rows per CTA with two CTAs per SM; else one.
    const bool two = 4 * row_bytes <= (size_t)maxsm;
    const int threads = 512;
    const size_t smem4 = (size_t)(zero_col(s->nsup) + kZeroCols) * 16;
    if (sizeof(T) == 4 && smem4 <= (size_t)maxsm) {
        // four rows per 1024-thread CTA, staged as 16-byte columns
        const size_t smem = smem4;
        int64_t blocks = (s->nsdn + 3) / 4;
        if (blocks > nsm) blocks = nsm;
        auto *kfn = a.ell_sg32 ? hub_row_col4_kernel<true> : hub_row_col4_kernel<false>;
        ED_CHECK_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kfn<<<(unsigned)blocks, 1024, smem, st>>>(reinterpret_cast<const float *>(x), reinterpret_cast<float *>(y), a);
    } else {
        const int R = two ? 2 : 1;
        const size_t smem = (size_t)R * row_bytes;
        auto *kfn = two ? hub_row_kernel<T, 2, false> : hub_row_kernel<T, 1, false>;
        if (sizeof(T) == 4 && a.ell_sg32) kfn = two ? hub_row_kernel<T, 2, sizeof(T) == 4> : hub_row_kernel<T, 1, sizeof(T) == 4>;
        ED_CHECK_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        // a warp per slice of short rows, and more CTAs: idle warps hold an SM's threads (18 sites (2,7), 5
        // slices, FP64 256 -> 199 us)
        const int nt = (int)std::min<int64_t>(threads, std::max<int64_t>(64, s->up.nslice * 32));
        const int64_t blocks = std::min<int64_t>((s->nsdn + R - 1) / R, (int64_t)nsm * (1024 / nt));
        kfn<<<(unsigned)blocks, nt, smem, st>>>(x, y, a, sld, vec_ok ? 1 : 0);
    }
    ED_CHECK_LAUNCH();
    // ---- the U_ijkl terms, if any (before pass 2, whose fused dots need the whole product)
    if (s->uijkl) {
        const int rc = uijkl_hv(s, st, sizeof(T) == 4 ? ED_F32 : ED_F64, ld, x, y, scale);
        if (rc != ED_OK) return rc;
    }
    // ---- pass 2
    // slab width: the x slab (nsdn rows x width) should take at most slab_l2_bytes() of L2
    int64_t slab_w = (int64_t)(slab_l2_bytes() / ((double)s->nsdn * sizeof(T)));
    slab_w = slab_w / 256 * 256;
    if (slab_w < 256) slab_w = 256;
    if (slab_w > s->nsup) slab_w = (s->nsup + VWS - 1) / VWS * VWS;
    const int64_t ngroups = (s->nsdn + 7) / 8;
    const bool vec2 = (ld % VWS == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0) &&
                      ((reinterpret_cast<uintptr_t>(y) & 15) == 0);
    // chunks x rows in flight, measured (4x4 slab pass / 14 random bonds): FP32 2 x 2 1,012 us / 148 us the
    // whole product, 1 x 4 1,070 / 154, 4 x 2 1,790 / 250 (registers); FP64 4 x 2 5.37 ms / 742 us, 2 x 4 6.26 / 743
    constexpr int U = sizeof(T) == 4 ? 2 : 4, kPass = 32 * VWS * U;
    // A pass of U chunks is 256 columns.  Rows with a good part of their columns past the whole passes take
    // those by single chunks: a column per lane there has one scalar load per hop and lane in flight (12 sites
    // (4,6), 495 strings, FP32 15.6 -> 9.6 us; half filled, 924 strings, 13.9 -> 11.1).  Where that part is small
    // (below a sixteenth) the two kernels are level.
    const bool single = s->nsup % kPass >= 32 && 16 * (s->nsup % kPass) >= s->nsup;
    auto *kfn = !vec2 ? hub_slab_kernel<T, 1, 1, 4, false>
                      : single ? hub_slab_kernel<T, VWS, U, 2, true> : hub_slab_kernel<T, VWS, U, 2, false>;
    // one wave of resident CTAs: each walks its share of the items, so a grid past the
    // resident count would leave a second, partial wave running whole shares
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, 256, 0);
    if (per_sm < 1) per_sm = 1;
    int64_t blocks2 = (int64_t)nsm * per_sm;
    if (blocks2 > kMaxPartialBlocks) blocks2 = kMaxPartialBlocks;
    // narrower slabs where a CTA's share would be a few items (the last of them would leave a part of
    // the wave idle: 14 sites FP32 160 -> 148 us)
    while (slab_w > 256 && ngroups * ((s->nsup + slab_w - 1) / slab_w) < 8 * blocks2)
        slab_w = std::max<int64_t>(256, slab_w / 2 / 256 * 256);
    const int64_t nslab = (s->nsup + slab_w - 1) / slab_w;
    const int64_t nitems = ngroups * nslab;
    if (blocks2 > nitems) blocks2 = nitems;
    if (blocks2 < 1) blocks2 = 1;
    double *part = dots ? partials : nullptr;
    kfn<<<(unsigned)blocks2, 256, 0, st>>>(x, y, a, (int)slab_w, (int)ngroups, (int)nitems, part);
    ED_CHECK_LAUNCH();
    if (dots) return launch_reduce(partials, (int)blocks2, 2, dots, st);
    return ED_OK;
}

}  // namespace ed

using namespace ed;

extern "C" int64_t ed_scratch_bytes(int64_t n, int nvec)
{
    (void)n;
    if (nvec < 1) nvec = 1;
    return (int64_t)kMaxPartialBlocks * 2 * nvec * (int64_t)sizeof(double) + 4096;
}

extern "C" int ed_hv_launches(const ed_sector *s, int dtype)
{
    if (!s || (dtype != ED_F32 && dtype != ED_F64)) return -1;
    if (s->dim == 0) return 0;
    if (s->kind != ED_HUBBARD) return 2;
    const bool one = dtype == ED_F32 ? one_pass<float>(s) : one_pass<double>(s);
    return (one ? 1 : 2) + (s->uijkl ? 1 : 0);
}

extern "C" int ed_hv(ed_sector *s, void *stream, int dtype, int64_t ld, const void *x, void *y, double scale,
                     double *dots, void *scratch, int64_t scratch_bytes)
{
    clear_error();
    ED_REQUIRE(s != nullptr, "sector is NULL");
    ED_REQUIRE(x != nullptr && y != nullptr, "x or y is NULL");
    ED_REQUIRE(x != y, "x and y must not alias");
    ED_REQUIRE(dtype == ED_F32 || dtype == ED_F64, "dtype must be ED_F32 or ED_F64");
    if (dots) {
        ED_REQUIRE(scratch != nullptr, "dots requested without scratch");
        ED_REQUIRE(scratch_bytes >= ed_scratch_bytes(s->dim, 1), "scratch of %lld bytes is below the %lld needed",
                   (long long)scratch_bytes, (long long)ed_scratch_bytes(s->dim, 1));
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (s->dim == 0) return ED_OK;
    if (s->kind == ED_HUBBARD) {
        ED_REQUIRE(ld >= s->nsup, "ld=%lld below nsup=%lld", (long long)ld, (long long)s->nsup);
        if (dtype == ED_F32)
            return hub_hv<float>(s, st, ld, static_cast<const float *>(x), static_cast<float *>(y), scale, dots,
                                 static_cast<double *>(scratch));
        return hub_hv<double>(s, st, ld, static_cast<const double *>(x), static_cast<double *>(y), scale, dots,
                              static_cast<double *>(scratch));
    }
    return heis_struct_hv(s, st, dtype, x, y, scale, dots, static_cast<double *>(scratch));
}
