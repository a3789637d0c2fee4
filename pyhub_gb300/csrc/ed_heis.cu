// ed_heis.cu -- structured H*v of the Heisenberg sector.
//
// Replaces HPROD of hprod_heis.f90:1-61 (the same Hamiltonian as heis_kernel
// of ed_hv.cu, element for element) with a product that never ranks a full
// 32-bit state.  A state is its empty-site (down-spin) pattern h, bit j for
// site j+1.  Split the sites into A = 1..nA (bits 0..nA-1) and B = the rest.
// The reference order is colex order of h, and colex order keeps all states
// that share their B part contiguous, ordered by the colex rank of their A
// part.  So the sector vector IS a set of rows: one row per B pattern hB
// (row offset = the colex contribution of hB's bits), and the row's entries
// are the A patterns with m = H - popcount(hB) holes in colex order (the
// 16-site combination order for a 4x8 lattice cut in two 4x4 halves).
// With that layout
//   A-A bonds flip within a row     -> gathers from the row staged in shared memory,
//   B-B bonds flip between rows     -> row axpys at equal column (coalesced),
//   A-B bonds flip both             -> a gather from ONE other row per bond; the
//                                      column map (add/remove one fixed bit) is
//                                      monotone, so the gathers stay local.
// Pass R (one CTA per row): diagonal + A-A + A-B, y = s*(...).
// Pass S (column slabs that keep the x slab of one m-block in L2): y += s*B-B,
// with the fused <x,y>, <y,y> partials.
#include "ed_common.cuh"

#include <cstdlib>

#include <algorithm>
#include <cstring>
#include <vector>

namespace ed {

namespace {

int64_t hbinom(int n, int k)
{
    if (k < 0 || n < 0 || k > n) return 0;
    int64_t r = 1;
    for (int i = 1; i <= k; ++i) r = r * (n - k + i) / i;
    return r;
}

// colex rank of a hole pattern: sum over its set bits p (ascending, i = 1..) of C(p, i)
int64_t colex_rank(uint32_t h, int base_i = 0, int shift = 0)
{
    int64_t r = 0;
    int i = base_i;
    while (h) {
        const int p = __builtin_ctz(h);
        r += hbinom(p + shift, ++i);
        h &= h - 1;
    }
    return r;
}

template <typename T>
int up(T **dst, const std::vector<T> &v)
{
    *dst = nullptr;
    if (v.empty()) return ED_OK;
    if (cudaMalloc(dst, sizeof(T) * v.size()) != cudaSuccess) {
        cudaGetLastError();
        set_error("device allocation of %zu bytes failed", sizeof(T) * v.size());
        return ED_ERR_MEM;
    }
    if (cudaMemcpy(*dst, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
        set_error("upload failed");
        return ED_ERR_CUDA;
    }
    return ED_OK;
}

}  // namespace

// Vectors up to this many bytes take orders that scatter reads and writes (FP64 columns by number of flips,
// rows by length): above it the scattered sectors come from DRAM more than once.  Several times the L2 (129 MB);
// the line lies between measured sizes: 29 sites (620 MB) 6.47 ms sorted, 6.67 in order; 30 (1.24 GB) 20.4, 14.0.
constexpr double kL2Bytes = 1.0e9;

int heis_struct_build(ed_sector *s)
{
    const HeisTables &ht = s->heis;
    HeisStruct *hs = new HeisStruct();
    s->hs = hs;
    const int norb = s->norb;
    const int nA = norb / 2, nB = norb - nA, H = norb - s->nup;
    hs->nA = nA;
    hs->nB = nB;
    hs->H = H;
    hs->mlo = std::max(0, H - nB);
    hs->mhi = std::min(nA, H);
    // ---- columns: A patterns by hole count m, colex order
    std::vector<uint32_t> col_pat;
    std::vector<int32_t> rankA((size_t)1 << nA, -1);
    std::vector<double> diagA;
    for (int m = 0; m <= kMaxHalf + 1; ++m) hs->col_base[m] = 0;
    for (int m = 0; m <= nA; ++m) {
        hs->col_base[m] = (int64_t)col_pat.size();
        hs->ncol[m] = hbinom(nA, m);
        std::vector<uint32_t> pats;
        for (uint32_t h = 0; h < (1u << nA); ++h)
            if (__builtin_popcount(h) == m) pats.push_back(h);
        std::sort(pats.begin(), pats.end(), [](uint32_t x, uint32_t y) { return colex_rank(x) < colex_rank(y); });
        for (size_t r = 0; r < pats.size(); ++r) {
            rankA[pats[r]] = (int32_t)r;
            col_pat.push_back(pats[r]);
        }
    }
    hs->col_base[nA + 1] = (int64_t)col_pat.size();
    // bonds by class
    std::vector<int> aa, bb, ab;
    for (int b = 0; b < ht.nbond; ++b) {
        const int pj = ht.bj[b] - 1, pk = ht.bk[b] - 1;   // pj < pk
        if (pk < nA) aa.push_back(b);
        else if (pj >= nA) bb.push_back(b);
        else ab.push_back(b);
    }
    if ((int)ab.size() > kMaxAB) {
        set_error("%zu bonds cross the two halves (at most %d)", ab.size(), kMaxAB);
        return ED_ERR_RANGE;
    }
    // A-A zz energy and hop lists per column, sliced ELL per m (32 columns per slice)
    diagA.resize(col_pat.size());
    std::vector<int32_t> aa_off(1, 0), aa64_off(1, 0), aa64_src, aa64_col;
    std::vector<int2> aa_pk32;
    std::vector<double> aa64_cf;
    int64_t nslices = 0;
    for (int m = 0; m <= nA; ++m) {
        hs->slice_base[m] = nslices;
        const int64_t n = hs->ncol[m], base = hs->col_base[m];
        std::vector<std::vector<std::pair<int32_t, double>>> lists((size_t)n);
        for (int64_t r = 0; r < n; ++r) {
            const uint32_t h = col_pat[(size_t)(base + r)];
            double d = 0.0;
            for (int b : aa) {
                const int pj = ht.bj[b] - 1, pk = ht.bk[b] - 1;
                const uint32_t hj = (h >> pj) & 1u, hk = (h >> pk) & 1u;
                d += (hj == hk ? 0.25 : -0.25) * ht.zz[b];
                if (hj == hk) continue;
                const double c = hj ? ht.flip_jk[b] : ht.flip_kj[b];
                if (c == 0.0) continue;
                lists[(size_t)r].push_back({rankA[h ^ ((1u << pj) | (1u << pk))], c});
            }
            diagA[(size_t)(base + r)] = d;
        }
        const int64_t ns = (n + 31) / 32;
        std::vector<int32_t> order((size_t)n);
        for (int64_t r = 0; r < n; ++r) order[(size_t)r] = (int32_t)r;
        // slots of the class, lane l of slice s with column order[s * 32 + l]; put(column, flip or NULL)
        auto slots = [&](std::vector<int32_t> &off, auto put) {
            for (int64_t sl = 0; sl < ns; ++sl) {
                size_t w = 0;
                for (int64_t r = sl * 32; r < std::min(n, sl * 32 + 32); ++r)
                    w = std::max(w, lists[(size_t)order[(size_t)r]].size());
                for (size_t k = 0; k < w; ++k)
                    for (int l = 0; l < 32; ++l) {
                        const int32_t c = order[(size_t)std::min(n - 1, sl * 32 + l)];
                        const auto &L = lists[(size_t)c];
                        put(c, sl * 32 + l < n && k < L.size() ? &L[k] : nullptr);   // none: own column, weight 0
                    }
                off.push_back(off.back() + (int32_t)w);
            }
        };
        slots(aa_off, [&](int32_t c, const std::pair<int32_t, double> *flip) {
            const float f = flip ? (float)flip->second : 0.f;
            int32_t bits;
            std::memcpy(&bits, &f, sizeof(bits));
            aa_pk32.push_back(make_int2(flip ? flip->first : c, bits));
        });
        // FP64: columns by number of flips.  A slice has as many slots as its longest list and each costs the
        // FP64 pipe a warp's operation (4x6: 12.9 slots for 9.4 flips in order, 9.7 by number), which
        // outweighs the scattered sources and results (row pass 140 -> 128 us, in windows of 128 132 us;
        // 4x7 3.41 -> 3.19 ms the whole product).  Vectors far above L2 pay for the scattering in DRAM
        // sectors (5x6, 1.2 GB: 14.9 -> 22.9 ms; 4x8 56 -> 78): windows of 64 there (14.9, 55.7 ms)
        const int64_t window = (double)s->dim * sizeof(double) <= kL2Bytes ? n : 64;
        for (int64_t r = 0; n > 32 && r < n; r += window)      // one slice: in order (the kernel relies on it)
            std::stable_sort(order.begin() + r, order.begin() + std::min(n, r + window), [&](int32_t x, int32_t y) {
                return lists[(size_t)x].size() > lists[(size_t)y].size();
            });
        slots(aa64_off, [&](int32_t c, const std::pair<int32_t, double> *flip) {
            aa64_src.push_back(flip ? flip->first : c);
            aa64_cf.push_back(flip ? flip->second : 0.0);
        });
        for (int64_t q = 0; q < ns * 32; ++q) aa64_col.push_back(q < n ? order[(size_t)q] : -1);
        nslices += ns;
    }
    hs->slice_base[nA + 1] = nslices;
    // ---- rows: B patterns with H - m holes, m in [mlo, mhi], sorted by offset
    struct Row {
        uint32_t hb;
        int m;
        int64_t off;
    };
    std::vector<Row> rows;
    for (uint32_t hb = 0; hb < (1u << nB); ++hb) {
        const int m = H - __builtin_popcount(hb);
        if (m < hs->mlo || m > hs->mhi) continue;
        // colex contribution of the B holes: running index continues after the m A holes
        rows.push_back({hb, m, colex_rank(hb, m, nA)});
    }
    std::sort(rows.begin(), rows.end(), [](const Row &x, const Row &y) { return x.off < y.off; });
    const int64_t nrows = (int64_t)rows.size();
    hs->nrows = nrows;
    std::vector<uint32_t> row_pat((size_t)nrows);
    std::vector<int32_t> row_m((size_t)nrows), rowidx((size_t)1 << nB, -1);
    std::vector<int64_t> row_off((size_t)nrows);
    std::vector<double> diagB((size_t)nrows);
    int64_t expect = 0;
    hs->max_len = 0;
    for (int64_t r = 0; r < nrows; ++r) {
        const Row &w = rows[(size_t)r];
        if (w.off != expect) {
            set_error("internal: row offsets are not contiguous at row %lld", (long long)r);
            return ED_ERR_ARG;
        }
        expect += hs->ncol[w.m];
        row_pat[(size_t)r] = w.hb;
        row_m[(size_t)r] = w.m;
        row_off[(size_t)r] = w.off;
        rowidx[w.hb] = (int32_t)r;
        hs->max_len = std::max<int64_t>(hs->max_len, hs->ncol[w.m]);
    }
    if (expect != s->nsup) {
        set_error("internal: rows cover %lld of %lld states", (long long)expect, (long long)s->nsup);
        return ED_ERR_ARG;
    }
    // A-B bonds: with at most 32 of them, a column's A bits and a row's B bits at the bonds are
    // packed into one word each; the bonds where they differ are the antiparallel ones
    hs->ab_fast = ab.size() <= 32;
    double ab_zz_sum = 0.0;   // sum of zz/4 over the A-B bonds (every bond taken as "equal")
    for (int b : ab) ab_zz_sum += 0.25 * ht.zz[b];
    std::vector<uint32_t> col_abbits, row_bbits;
    std::vector<double> ab_lut;
    std::vector<int32_t> ab_rank;   // [q][column]: rank of the column's pattern with the bond's A bit flipped
    if (hs->ab_fast) {
        ab_rank.resize(ab.size() * col_pat.size());
        for (size_t q = 0; q < ab.size(); ++q)
            for (size_t c = 0; c < col_pat.size(); ++c)
                ab_rank[q * col_pat.size() + c] = rankA[col_pat[c] ^ (1u << (ht.bj[ab[q]] - 1))];
        hs->ncols = (int64_t)col_pat.size();
        ab_lut.assign(4 * 256, 0.0);      // also without A-B bonds: the kernels always look the first eight up
        for (size_t k = 0; k < ab_lut.size(); ++k)
            for (size_t q = 0; q < 8; ++q) {
                const size_t bond = k / 256 * 8 + q;
                if (bond < ab.size() && ((k >> q) & 1)) ab_lut[k] += 0.5 * ht.zz[ab[bond]];
            }
        col_abbits.resize(col_pat.size());
        for (size_t c = 0; c < col_pat.size(); ++c) {
            uint32_t w = 0;
            for (size_t q = 0; q < ab.size(); ++q) w |= ((col_pat[c] >> (ht.bj[ab[q]] - 1)) & 1u) << q;
            col_abbits[c] = w;
        }
        row_bbits.resize((size_t)nrows);
        for (int64_t r = 0; r < nrows; ++r) {
            uint32_t w = 0;
            for (size_t q = 0; q < ab.size(); ++q) w |= ((row_pat[(size_t)r] >> (ht.bk[ab[q]] - 1 - nA)) & 1u) << q;
            row_bbits[(size_t)r] = w;
        }
    }
    // B-B zz energy (+ the constant diagonal) and neighbour rows per row
    std::vector<int32_t> bb_ptr(1, 0), bb_src;
    std::vector<double> bb_cf;
    for (int64_t r = 0; r < nrows; ++r) {
        const uint32_t h = row_pat[(size_t)r];
        double d = ht.dconst + (hs->ab_fast ? ab_zz_sum : 0.0);
        for (int b : bb) {
            const int pj = ht.bj[b] - 1 - nA, pk = ht.bk[b] - 1 - nA;
            const uint32_t hj = (h >> pj) & 1u, hk = (h >> pk) & 1u;
            d += (hj == hk ? 0.25 : -0.25) * ht.zz[b];
            if (hj == hk) continue;
            const double c = hj ? ht.flip_jk[b] : ht.flip_kj[b];
            if (c == 0.0) continue;
            bb_src.push_back(rowidx[h ^ ((1u << pj) | (1u << pk))]);
            bb_cf.push_back(c);
        }
        diagB[(size_t)r] = d;
        bb_ptr.push_back((int32_t)bb_src.size());
    }
    // rows grouped by m (offset order within each m) for the slab pass
    std::vector<int32_t> rows_of_m;
    for (int m = 0; m <= kMaxHalf + 1; ++m) hs->row_base[m] = 0;
    for (int m = 0; m <= nA; ++m) {
        hs->row_base[m] = (int64_t)rows_of_m.size();
        for (int64_t r = 0; r < nrows; ++r)
            if (row_m[(size_t)r] == m) rows_of_m.push_back((int32_t)r);
    }
    hs->row_base[nA + 1] = (int64_t)rows_of_m.size();
    // A-B bonds
    hs->nab = (int)ab.size();
    for (int q = 0; q < hs->nab; ++q) {
        const int b = ab[(size_t)q];
        hs->ab_pa[q] = (int8_t)(ht.bj[b] - 1);
        hs->ab_pb[q] = (int8_t)(ht.bk[b] - 1 - nA);
        hs->ab_fjk[q] = ht.flip_jk[b];
        hs->ab_fkj[q] = ht.flip_kj[b];
        hs->ab_zz[q] = 0.25 * ht.zz[b];
    }
    std::vector<float> ab_lut32(ab_lut.begin(), ab_lut.end());
    std::vector<float> bb_cf32(bb_cf.begin(), bb_cf.end());
    std::vector<float> diagA32(diagA.begin(), diagA.end()), diagB32(diagB.begin(), diagB.end());
    int rc;
    if ((rc = up(&hs->col_pat, col_pat)) || (rc = up(&hs->rankA, rankA)) || (rc = up(&hs->diagA, diagA)) ||
        (rc = up(&hs->aa_off, aa_off)) || (rc = up(&hs->aa64_off, aa64_off)) ||
        (rc = up(&hs->aa64_src, aa64_src)) || (rc = up(&hs->aa64_col, aa64_col)) || (rc = up(&hs->aa64_cf, aa64_cf)) ||
        (rc = up(&hs->row_pat, row_pat)) || (rc = up(&hs->row_m, row_m)) ||
        (rc = up(&hs->row_off, row_off)) || (rc = up(&hs->rowidx, rowidx)) || (rc = up(&hs->diagB, diagB)) ||
        (rc = up(&hs->bb_ptr, bb_ptr)) || (rc = up(&hs->bb_src, bb_src)) || (rc = up(&hs->bb_cf32, bb_cf32)) ||
        (rc = up(&hs->bb_cf64, bb_cf)) || (rc = up(&hs->rows_of_m, rows_of_m)) ||
        (rc = up(&hs->aa_pk32, aa_pk32)) || (rc = up(&hs->col_abbits, col_abbits)) ||
        (rc = up(&hs->row_bbits, row_bbits)) || (rc = up(&hs->diagA32, diagA32)) || (rc = up(&hs->ab_rank, ab_rank)) ||
        (rc = up(&hs->diagB32, diagB32)) || (rc = up(&hs->ab_lut, ab_lut)) || (rc = up(&hs->ab_lut32, ab_lut32)))
        return rc;
    return ED_OK;
}

void heis_struct_free(HeisStruct *hs)
{
    if (!hs) return;
    void *ptrs[] = {hs->col_pat, hs->rankA, hs->diagA, hs->aa_off, hs->aa64_off, hs->aa64_src,
                    hs->aa64_col, hs->aa64_cf, hs->row_pat, hs->row_m, hs->row_off, hs->rowidx, hs->diagB,
                    hs->bb_ptr, hs->bb_src, hs->bb_cf32, hs->bb_cf64, hs->rows_of_m,
                    hs->aa_pk32, hs->col_abbits, hs->row_bbits, hs->diagA32, hs->diagB32, hs->ab_rank,
                    hs->ab_lut, hs->ab_lut32};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    delete hs;
}

// ------------------------------------------------------------ kernels

struct HsArgs {
    int nA, nB, nab;
    int64_t nrows;
    int64_t col_base[kMaxHalf + 2], ncol[kMaxHalf + 1], slice_base[kMaxHalf + 2], row_base[kMaxHalf + 2];
    const uint32_t *col_pat, *row_pat;
    const int32_t *rankA, *aa_off, *aa64_src, *aa64_col, *row_m, *rowidx, *bb_ptr, *bb_src, *rows_of_m;
    const int64_t *row_off;
    const void *diagA, *diagB;     // float or double, like the vectors
    const void *bb_cf;             // float or double
    const int2 *aa_pk32;           // {column, FP32 coefficient bits} of the A-A flips
    const double *aa64_cf;
    const uint32_t *col_abbits, *row_bbits;
    const int32_t *ab_rank;        // [q][column] rank after flipping bond q's A bit (packed path)
    const void *ab_lut;            // [4][256] zz drops of eight bonds, float or double
    int64_t ncols;
    int ab_fast;
    int8_t ab_pa[kMaxAB], ab_pb[kMaxAB];
    double ab_fjk[kMaxAB], ab_fkj[kMaxAB], ab_zz[kMaxAB];
    double scale;
    int8_t m_order[kMaxHalf + 1];  // the hole counts of A by falling row length
    int by_length;                 // one-row pass: rows in that order, else in the vector's
};

// Work item `at` of a CTA's walk in round k: rounds alternate in direction over items sorted by falling
// length, so that the CTAs' sums of lengths stay close.
__device__ __forceinline__ int64_t zigzag(int64_t k)
{
    return k * gridDim.x + ((k & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
}

constexpr int kHeisRowThreads = 512;

// bytes of the A-B bond facts ahead of the staged row (16-byte aligned)
__host__ __device__ inline size_t heis_row_head_bytes(int nab, size_t tsize)
{
    const size_t b = (size_t)nab * (sizeof(int64_t) + 2 * tsize + sizeof(uint32_t));
    return (b + 15) / 16 * 16;
}
constexpr int64_t kMaxPartialBlocksHeis = 1024;   // the partials that ed_scratch_bytes provides for

// Pass R: y[row] = s * (diag + A-A flips + A-B flips) of every row.
template <typename T>
__global__ void __launch_bounds__(kHeisRowThreads, 4) heis_row_kernel(const T *__restrict__ x, T *__restrict__ y,
                                                                    const HsArgs a)
{
    // dynamic shared memory: per-row A-B bond facts (nab entries each), then the staged row
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int64_t *ab_src = reinterpret_cast<int64_t *>(smem_raw);      // source row offset, -1 if impossible
    T *ab_c = reinterpret_cast<T *>(ab_src + a.nab);               // flip element for the required A state
    T *ab_dsame = ab_c + a.nab;                                    // zz/4 (generic path)
    uint32_t *ab_need = reinterpret_cast<uint32_t *>(ab_dsame + a.nab);  // required A bit (1: A site down)
    T *xs = reinterpret_cast<T *>(smem_raw + heis_row_head_bytes(a.nab, sizeof(T)));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = kHeisRowThreads / 32;
    const T sc = (T)a.scale;
    for (int64_t k = 0; k * gridDim.x < a.nrows; ++k) {
        int m;
        int64_t row;
        if (a.by_length) {
            int64_t g = zigzag(k);
            if (g >= a.nrows) continue;
            int o = 0;
            m = a.m_order[0];
            for (;;) {
                const int64_t nr_m = a.row_base[m + 1] - a.row_base[m];
                if (g < nr_m) break;
                g -= nr_m;
                m = a.m_order[++o];
            }
            row = __ldg(a.rows_of_m + a.row_base[m] + g);
        } else {
            row = k * gridDim.x + blockIdx.x;
            if (row >= a.nrows) continue;
            m = __ldg(a.row_m + row);
        }
        const uint32_t hb = __ldg(a.row_pat + row);
        const int64_t off = __ldg(a.row_off + row);
        const int len = (int)a.ncol[m];
        const int64_t cbase = a.col_base[m];
        const int64_t sbase = a.slice_base[m];
        const T db = __ldg(static_cast<const T *>(a.diagB) + row);
        const uint32_t rbits = a.ab_fast ? __ldg(a.row_bbits + row) : 0u;
        __syncthreads();   // the previous row's readers are done with xs / ab_*
        // asynchronous copies: the whole row in flight at once
        for (int c = threadIdx.x; c < len; c += blockDim.x) cp_async_elem(xs + c, x + off + c);
        for (int q = threadIdx.x; q < a.nab; q += blockDim.x) {
            const uint32_t hk = (hb >> a.ab_pb[q]) & 1u;
            // the flip needs the A site opposite to the B site: hj = 1 - hk
            const int32_t r2 = __ldg(a.rowidx + (hb ^ (1u << a.ab_pb[q])));
            ab_src[q] = (r2 >= 0) ? __ldg(a.row_off + r2) : (int64_t)-1;
            ab_need[q] = 1u - hk;
            ab_c[q] = (T)(hk ? a.ab_fkj[q] : a.ab_fjk[q]);   // target hj = 1-hk: hj ? fjk : fkj
            ab_dsame[q] = (T)a.ab_zz[q];
        }
        cp_async_wait_all();
        __syncthreads();
        const int nsl = (len + 31) / 32;
        for (int sl = warp; sl < nsl; sl += nwarps) {
            // (a class of one slice is in order, and the look-up would lead a short row's chain of loads)
            const bool plain = sizeof(T) == 4 || len <= 32;
            const int c = plain ? sl * 32 + lane : __ldg(a.aa64_col + (sbase + sl) * 32 + lane);
            const bool ok = plain ? c < len : c >= 0;
            const int cc = ok ? c : len - 1;
            const uint32_t ha = __ldg(a.col_pat + cbase + cc);
            T d = __ldg(static_cast<const T *>(a.diagA) + cbase + cc) + db;
            T acc = 0;
            const int s0 = __ldg(a.aa_off + sbase + sl), ns = __ldg(a.aa_off + sbase + sl + 1) - s0;
            // antiparallel A-B bonds: the set bits of (column's A bits ^ row's B bits); their zz/4 was counted
            // as "equal" in diagB, so each one drops the diagonal by zz/2.  Eight bonds' drops come from a
            // table; the first look-up is in flight during the A-A flips
            const T *lut = static_cast<const T *>(a.ab_lut);
            uint32_t diff = 0u;
            T drop = 0;
            if (a.ab_fast) {
                diff = __ldg(a.col_abbits + cbase + cc) ^ rbits;
                drop = __ldg(lut + (diff & 255u));
            }
            if (sizeof(T) == 4) {
#pragma unroll 4
                for (int q = 0; q < ns; ++q) {
                    const int2 pk = __ldg(a.aa_pk32 + (s0 + q) * 32 + lane);
                    acc += (T)__int_as_float(pk.y) * xs[pk.x];
                }
            } else {
#pragma unroll 4
                for (int q = 0; q < ns; ++q) {
                    const int at = (s0 + q) * 32 + lane;
                    acc += (T)__ldg(a.aa64_cf + at) * xs[__ldg(a.aa64_src + at)];
                }
            }
            if (a.ab_fast) {
                d -= drop;
                for (int g = 1; g * 8 < a.nab; ++g) d -= __ldg(lut + g * 256 + ((diff >> (8 * g)) & 255u));
                while (diff) {
                    const int q = __ffs(diff) - 1;
                    diff &= diff - 1;
                    const int64_t src = ab_src[q];
                    if (src >= 0) acc += ab_c[q] * __ldg(x + src + __ldg(a.ab_rank + q * a.ncols + cbase + cc));
                }
            } else
            for (int q = 0; q < a.nab; ++q) {
                const uint32_t hj = (ha >> a.ab_pa[q]) & 1u;
                if (hj != ab_need[q]) {
                    d += ab_dsame[q];          // equal sites
                    continue;
                }
                d -= ab_dsame[q];
                const int64_t src = ab_src[q];
                if (src >= 0) acc += ab_c[q] * __ldg(x + src + __ldg(a.rankA + (ha ^ (1u << a.ab_pa[q]))));
            }
            const T v = d * xs[cc] + acc;
            if (ok) y[off + c] = (sc == (T)1) ? v : v * sc;
        }
    }
}

constexpr int kHeisCol4Threads = 1024;

// An A-B bond of one staged row: the source row's first element (a sector has fewer than 2^31) and the
// flip element.  A column antiparallel to the row at the bond always has that row.
struct alignas(8) AbFact {
    int src;
    float c;
};

// bytes of the four rows' A-B bond facts ahead of the staged columns (16-byte aligned)
__host__ __device__ inline size_t heis_col4_head_bytes(int nab)
{
    const size_t b = (size_t)nab * 4 * sizeof(AbFact);
    return (b + 15) / 16 * 16;
}

// G A-A flip slots of one lane (table entries at, at+32, ...) applied to the
// four staged rows; the G table loads are issued before the first gather.
template <int G>
__device__ __forceinline__ void heis_col4_group(const HsArgs &a, int at, const float4 *xs4, float (&acc)[4])
{
    int q[G];
    float c[G];
#pragma unroll
    for (int i = 0; i < G; ++i) {
        const int2 pk = __ldg(a.aa_pk32 + at + i * 32);
        q[i] = pk.x;
        c[i] = __int_as_float(pk.y);
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

// Pass R for FP32 with four rows of one hole count per CTA (packed A-B path):
// the four rows' entries of column c are staged as one 16-byte column xs4[c],
// so one A-A flip slot (an 8-byte table load) and one 128-bit gather serve all
// four rows.  Each row's sums are the one-row kernel's, in its order (slots,
// then the antiparallel A-B bonds in increasing order), so the product is the same.
// Work items are groups of four rows of rows_of_m, hole count by hole count.
// Bound by the latency of its loads: the A-B bonds' dependent pair (rank of the
// flipped column, then the element) goes four bonds at a time, up to 16
// elements in flight (one bond at a time: 4x7 957 us, now 600); two CTAs per SM
// where their rows fit.
__global__ void __launch_bounds__(kHeisCol4Threads, 1) heis_row_col4_kernel(const float *__restrict__ x,
                                                                          float *__restrict__ y, const HsArgs a,
                                                                          int64_t nitems)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    AbFact *facts = reinterpret_cast<AbFact *>(smem_raw);          // [4][nab]
    float4 *xs4 = reinterpret_cast<float4 *>(smem_raw + heis_col4_head_bytes(a.nab));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const float sc = (float)a.scale;
    const float *dA32 = static_cast<const float *>(a.diagA), *dB32 = static_cast<const float *>(a.diagB);
    for (int64_t k = 0; k * gridDim.x < nitems; ++k) {
        int64_t g = zigzag(k);
        if (g >= nitems) continue;
        int o = 0, m = a.m_order[0];
        for (;;) {
            const int64_t ng = (a.row_base[m + 1] - a.row_base[m] + 3) / 4;
            if (g < ng) break;
            g -= ng;
            m = a.m_order[++o];
        }
        const int nr = (int)min((int64_t)4, a.row_base[m + 1] - a.row_base[m] - 4 * g);
        int64_t off[4];
        float db[4];
        uint32_t rbits[4], hb[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int32_t row = __ldg(a.rows_of_m + a.row_base[m] + 4 * g + (r < nr ? r : 0));
            off[r] = __ldg(a.row_off + row);
            db[r] = __ldg(dB32 + row);
            rbits[r] = __ldg(a.row_bbits + row);
            hb[r] = __ldg(a.row_pat + row);
        }
        const int len = (int)a.ncol[m];
        const int64_t cbase = a.col_base[m];
        const int64_t sbase = a.slice_base[m];
        __syncthreads();   // the previous group's readers are done with xs4 / ab_*
        for (int c = threadIdx.x; c < len; c += blockDim.x) {
            float *dst = reinterpret_cast<float *>(xs4 + c);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (r < nr) cp_async_elem(dst + r, x + off[r] + c);
                else dst[r] = 0.f;
            }
        }
        for (int t = threadIdx.x; t < 4 * a.nab; t += blockDim.x) {
            const int r = t / a.nab, q = t - r * a.nab;
            AbFact f = {0, 0.f};
            if (r < nr) {
                const uint32_t h = (r == 0) ? hb[0] : (r == 1) ? hb[1] : (r == 2) ? hb[2] : hb[3];
                const uint32_t hk = (h >> a.ab_pb[q]) & 1u;
                const int32_t r2 = __ldg(a.rowidx + (h ^ (1u << a.ab_pb[q])));
                if (r2 >= 0) {
                    f.src = (int)__ldg(a.row_off + r2);
                    f.c = (float)(hk ? a.ab_fkj[q] : a.ab_fjk[q]);
                }
            }
            facts[t] = f;
        }
        cp_async_wait_all();
        __syncthreads();
        const int nsl = (len + 31) / 32;
        for (int sl = warp; sl < nsl; sl += nwarps) {
            const int c = sl * 32 + lane;
            const bool ok = c < len;
            const int cc = ok ? c : len - 1;
            const float dA = __ldg(dA32 + cbase + cc);
            float d[4], acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int r = 0; r < 4; ++r) d[r] = dA + db[r];
            const int s0 = __ldg(a.aa_off + sbase + sl), ns = __ldg(a.aa_off + sbase + sl + 1) - s0;
            // slots in groups: all table loads of a group are in flight before its first gather
            const int at0 = s0 * 32 + lane;
            int q = 0;
            for (; q + 8 <= ns; q += 8) heis_col4_group<8>(a, at0 + q * 32, xs4, acc);
            if (q + 4 <= ns) {
                heis_col4_group<4>(a, at0 + q * 32, xs4, acc);
                q += 4;
            }
            for (; q < ns; ++q) heis_col4_group<1>(a, at0 + q * 32, xs4, acc);
            // antiparallel A-B bonds of each row: the set bits of (column's A bits ^ row's B bits)
            const uint32_t ca = __ldg(a.col_abbits + cbase + cc);
            const float *lut = static_cast<const float *>(a.ab_lut);
            uint32_t diff[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                diff[r] = (r < nr) ? (ca ^ rbits[r]) : 0u;
#pragma unroll
                for (int g8 = 0; g8 < 4; ++g8)
                    if (g8 * 8 < a.nab) d[r] -= __ldg(lut + g8 * 256 + ((diff[r] >> (8 * g8)) & 255u));
            }
            // four bonds at a time: their ranks, then their up to 16 source elements, are in flight together
            const int32_t *rank = a.ab_rank + cbase + cc;
            const int ncols = (int)a.ncols;     // at most 32 x 2^16 table entries
            for (int q0 = 0; q0 < a.nab; q0 += 4) {
                int rk[4];
                float v[4][4];
#pragma unroll
                for (int i = 0; i < 4; ++i) rk[i] = (q0 + i < a.nab) ? __ldg(rank + (q0 + i) * ncols) : 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (q0 + i >= a.nab) break;
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        v[i][r] = 0.f;
                        if ((diff[r] >> (q0 + i)) & 1u) v[i][r] = __ldg(x + (facts[r * a.nab + q0 + i].src + rk[i]));
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (q0 + i >= a.nab) break;
#pragma unroll
                    for (int r = 0; r < 4; ++r) acc[r] += facts[r * a.nab + q0 + i].c * v[i][r];
                }
            }
            if (ok) {
                const float4 xv = xs4[cc];
                const float xr[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (r < nr) y[off[r] + c] = (d[r] * xr[r] + acc[r]) * sc;
            }
        }
    }
}

// Pass S: y += s * (B-B flips), fused <x,y>, <y,y>.  Work items run block
// (m) by block, slab by slab: all row groups of a block read one column slab
// of x while it sits in L2.
struct SlabPlan {
    int nblk;
    int m[kMaxHalf + 1];
    int64_t item_base[kMaxHalf + 2];
    int64_t slab_w[kMaxHalf + 1], ngroups[kMaxHalf + 1];
};

constexpr int kHeisSlabCtas = 3;     // CTAs per SM: up to 80 registers a thread

template <typename T>
__global__ void __launch_bounds__(256, kHeisSlabCtas) heis_slab_kernel(const T *__restrict__ x, T *__restrict__ y,
                                                                       const HsArgs a, const SlabPlan p,
                                                                       double *__restrict__ partials)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const T *bcf = reinterpret_cast<const T *>(a.bb_cf);
    const T sc = (T)a.scale;
    double dxy = 0.0, dyy = 0.0;
    const int64_t nitems = p.item_base[p.nblk];
    for (int64_t it = blockIdx.x; it < nitems; it += gridDim.x) {
        int bi = 0;
        while (bi + 1 < p.nblk && p.item_base[bi + 1] <= it) ++bi;
        const int m = p.m[bi];
        const int64_t li = it - p.item_base[bi];
        const int64_t slab = li / p.ngroups[bi], g = li - slab * p.ngroups[bi];
        const int len = (int)a.ncol[m];
        const int64_t nr_m = a.row_base[m + 1] - a.row_base[m];
        const int64_t rr = g * 8 + warp;
        if (rr >= nr_m) continue;   // warp-uniform
        const int32_t row = __ldg(a.rows_of_m + a.row_base[m] + rr);
        const int64_t off = __ldg(a.row_off + row);
        const int e0 = __ldg(a.bb_ptr + row), nn = __ldg(a.bb_ptr + row + 1) - e0;
        const int64_t c0 = slab * p.slab_w[bi];
        const int64_t c1 = min((int64_t)len, c0 + p.slab_w[bi]);
        for (int eb = 0; eb < nn || eb == 0; eb += 32) {
            // neighbour rows of this chunk, one per lane
            const int ne = min(32, nn - eb);
            int64_t my_off = 0;
            T my_cf = 0;
            if (lane < ne) {
                my_off = __ldg(a.row_off + __ldg(a.bb_src + e0 + eb + lane));
                my_cf = __ldg(bcf + e0 + eb + lane);
            }
            const bool last = eb + 32 >= nn;
            T sxy = 0, syy = 0;
            // four 32-column chunks per pass.  Bound by L2 latency (rows start at any element, so a load is
            // 4 or 8 bytes per lane): a pass that lies inside the row issues the loads of G neighbour rows,
            // 4 G of them, before the first sum (4x7 FP32: 584 us with one row's loads, 274 with four rows').
            constexpr int G = sizeof(T) == 4 ? 4 : 2;
            int64_t cb = c0;
            for (; cb + 128 <= c1; cb += 128) {
                const T *xc = x + cb + lane;
                T *yc = y + off + cb + lane;
                T acc[4] = {0, 0, 0, 0}, yv[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) yv[j] = yc[32 * j];
                int e = 0;
                for (; e + G <= ne; e += G) {
                    T v[G][4], w[G];
#pragma unroll
                    for (int i = 0; i < G; ++i) {
                        const int64_t so = __shfl_sync(0xffffffffu, my_off, e + i);
                        w[i] = __shfl_sync(0xffffffffu, my_cf, e + i);
#pragma unroll
                        for (int j = 0; j < 4; ++j) v[i][j] = __ldg(xc + so + 32 * j);
                    }
#pragma unroll
                    for (int i = 0; i < G; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j) acc[j] += w[i] * v[i][j];
                }
                for (; e < ne; ++e) {
                    const int64_t so = __shfl_sync(0xffffffffu, my_off, e);
                    const T w = __shfl_sync(0xffffffffu, my_cf, e);
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[j] += w * __ldg(xc + so + 32 * j);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    yv[j] += acc[j] * sc;
                    yc[32 * j] = yv[j];
                    if (last && partials) {
                        sxy += x[off + cb + lane + 32 * j] * yv[j];
                        syy += yv[j] * yv[j];
                    }
                }
            }
            if (cb < c1) {
                T acc[4] = {0, 0, 0, 0};
#pragma unroll 2
                for (int e = 0; e < ne; ++e) {
                    const int64_t so = __shfl_sync(0xffffffffu, my_off, e);
                    const T w = __shfl_sync(0xffffffffu, my_cf, e);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int64_t c = cb + 32 * j + lane;
                        if (c < c1) acc[j] += w * __ldg(x + so + c);
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int64_t c = cb + 32 * j + lane;
                    if (c < c1) {
                        const T yv = y[off + c] + acc[j] * sc;
                        y[off + c] = yv;
                        if (last && partials) {
                            sxy += x[off + c] * yv;
                            syy += yv * yv;
                        }
                    }
                }
            }
            dxy += (double)sxy;
            dyy += (double)syy;
        }
    }
    if (partials) {
        __shared__ double red[2][8];
        dxy = warp_sum(dxy);
        dyy = warp_sum(dyy);
        if (lane == 0) {
            red[0][warp] = dxy;
            red[1][warp] = dyy;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double sxy = 0.0, syy = 0.0;
            for (int w = 0; w < 8; ++w) {
                sxy += red[0][w];
                syy += red[1][w];
            }
            partials[2 * blockIdx.x] = sxy;
            partials[2 * blockIdx.x + 1] = syy;
        }
    }
}

// ------------------------------------------------------------ spin correlations
//
// J_SPIN of the Heisenberg solver (static_rq_heis.f90:58-116) on the row
// layout, per pair p = (J,K) of the caller's list:
//   q[p][0] = J!=K: sum over states I with J up, K down of (-1)^(J+K) bra[I'] ket[I]
//             (I' = I with J and K swapped);  J==K: 0.5 sum bra ket
//   q[p][1] = sum bra ket Sz_J Sz_K
// Everything here is bound by the FP64 pipe (2 FMA per clock and SM), so the kernels enumerate the
// states that take part instead of testing all of them: a test leaves the other lanes' FP64 slots
// empty (26% of the states take part in a flip).  When bra is ket, q[(J,K)] and q[(K,J)] hold the
// same products (I <-> I') and are formed once.
//   * rdm_flips: a warp owns one task over one chunk of rows.  Two A sites: the columns
//     with J up, K down are the patterns of the other sites with one hole less, two bits inserted;
//     lanes over those columns, each applied to all the chunk's rows of that class.  Two B sites:
//     whole rows against their swapped rows.  An A site J and every B site asked for with it: the
//     columns with J fixed against one other row per B site, so an element of ket is loaded once
//     for all of them.
//   * rdm_diag_tile: the Sz Sz sums with an A site, factorised through column sums.
//   * rdm_rows: those of two B sites, from row sums.
// The three run as one launch.  All pairs of 24 sites, FP64, whole call: 6.38 ms with every ordered
// pair tested state by state and 31 FP64 operations per element of the diagonal sums, 0.69 ms in
// this form; 8 sites 69 -> 68 us, 16 sites 371 -> 125 us.  NB bounds the sites of the B half (the sums a
// lane keeps), CTAS the CTAs of an SM.

constexpr int kRdmTasks = kMaxSites * kMaxSites;
constexpr int kRdmChunks = 512;

struct HsRdmArgs {
    int nA, nB, npairs;
    int64_t col_base[kMaxHalf + 2], ncol[kMaxHalf + 1];
    const uint32_t *col_pat, *row_pat;
    const int32_t *rankA, *rowidx, *rows_of_m;
    const int64_t *row_off;
    int64_t row_base[kMaxHalf + 2];
    int8_t pj[kRdmTasks], pk[kRdmTasks];    // the distinct pairs: hole-bit positions (site-1)
    // flip tasks: nab pairs (A site, orientation) first, then one per pair of two A or two B sites
    int nab, ntask, nbb;
    int8_t ab_site[2 * kMaxHalf], ab_bit[2 * kMaxHalf];
    uint32_t ab_mask[2 * kMaxHalf];         // B sites asked for
    int16_t ab_pair[2 * kMaxHalf][kMaxHalf];
    int16_t task_pair[kRdmTasks], bb_pair[kRdmTasks];
    // rows in rows_of_m order are cut into chunks of about equal numbers of states
    int chunk0[kRdmChunks + 1];
    int tile_base[kMaxHalf + 2], nry[kMaxHalf + 1];   // tiles of the diagonal pass per class m
};

constexpr int kRdmThreads = 256;
// Sectors of this many states take five CTAs per SM instead of three: the flips wait for loads most of the
// time and more warps cover them, at the price of spilled registers, most of them in the diagonal tiles (all
// pairs, FP64, three and five: 20 sites, 184,756 states, 149 and 161 us; 21, 352,716, 219 and 200; 22 272 and 240;
// 24 709 and 627; FP32 168 and 174, 260 and 251, 343 and 330, 1,047 and 1,049; but the 21 bonds of a 21-site ring
// 173 and 185, so that sector keeps three).
constexpr int64_t kRdmLarge = 1 << 19;

__device__ __forceinline__ uint32_t insert_bit(uint32_t h, int pos, uint32_t bit)
{
    const uint32_t low = (1u << pos) - 1u;
    return (h & low) | ((h & ~low) << 1) | (bit << pos);
}

// acc + b k in FP64; FP32 vectors form the product in FP32, as their sums over a row always have
template <typename T> __device__ __forceinline__ void mul_add(double &acc, T b, T k)
{
    if constexpr (sizeof(T) == 8) acc = fma(b, k, acc);
    else acc += (double)(b * k);
}

template <typename T, int NB>
__device__ __forceinline__ void rdm_flips(const T *__restrict__ bra, const T *__restrict__ ket, const HsRdmArgs &a,
                                          int mlo, int mhi, int task, int chunk, double *__restrict__ partials)
{
    const int lane = threadIdx.x & 31;
    if (task >= a.ntask) return;
    double *out = partials + (int64_t)chunk * a.npairs * 2;
    const int64_t p0 = a.chunk0[chunk], p1 = a.chunk0[chunk + 1];
    if (task < a.nab) {
        const int J = a.ab_site[task];
        const uint32_t bit = (uint32_t)a.ab_bit[task], mask = a.ab_mask[task];
        double acc[NB];
#pragma unroll
        for (int k = 0; k < NB; ++k) acc[k] = 0.0;
        for (int m = mlo; m <= mhi; ++m) {
            const int64_t ra = max(p0, a.row_base[m]), rb = min(p1, a.row_base[m + 1]);
            if (ra >= rb || m < (int)bit) continue;
            // the patterns of the other nA - 1 A sites with m - bit holes are the first of their class
            const int hm = m - (int)bit;
            if (hm > a.nA - 1) continue;
            int64_t ne = 1;
            for (int i = 1; i <= hm; ++i) ne = ne * (a.nA - 1 - hm + i) / i;
            for (int64_t r = ra; r < rb; ++r) {
                const int32_t row = __ldg(a.rows_of_m + r);
                const uint32_t hb = __ldg(a.row_pat + row);
                const uint32_t need = mask & (bit ? ~hb : hb);
                if (!need) continue;
                const T *kr = ket + __ldg(a.row_off + row);
                int my_off = 0;      // a sector has fewer than 2^31 states
                if ((need >> lane) & 1u) my_off = (int)__ldg(a.row_off + __ldg(a.rowidx + (hb ^ (1u << lane))));
                for (int64_t e0 = 0; e0 < ne; e0 += 32) {
                    const int64_t e = e0 + lane;
                    const bool ok = e < ne;
                    const uint32_t base = __ldg(a.col_pat + a.col_base[hm] + (ok ? e : 0));
                    const uint32_t h = insert_bit(base, J, bit);
                    const int c = __ldg(a.rankA + h), c2 = __ldg(a.rankA + (h ^ (1u << J)));
                    const T kv = ok ? __ldg(kr + c) : (T)0;
#pragma unroll
                    for (int k = 0; k < NB; ++k) {
                        if ((need >> k) & 1u) {
                            const int o2 = __shfl_sync(0xffffffffu, my_off, k);
                            mul_add<T>(acc[k], __ldg(bra + o2 + c2), kv);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            if (!((mask >> k) & 1u)) continue;
            const double s = warp_sum(acc[k]);
            if (lane == 0) out[2 * a.ab_pair[task][k]] = ((J + k + a.nA) & 1) ? -s : s;
        }
        return;
    }
    const int p = a.task_pair[task - a.nab];
    const int J = a.pj[p], K = a.pk[p];
    double acc = 0.0;
    if (J < a.nA) {     // two A sites
        const int lo = min(J, K), hi = max(J, K);
        const uint32_t mask = (1u << J) | (1u << K);
        for (int m = max(mlo, 1); m <= mhi; ++m) {
            const int64_t ra = max(p0, a.row_base[m]), rb = min(p1, a.row_base[m + 1]);
            if (ra >= rb || m - 1 > a.nA - 2) continue;
            int64_t ne = 1;
            for (int i = 1; i <= m - 1; ++i) ne = ne * (a.nA - 2 - (m - 1) + i) / i;
            for (int64_t e = lane; e < ne; e += 32) {
                const uint32_t base = __ldg(a.col_pat + a.col_base[m - 1] + e);
                const uint32_t h = insert_bit(insert_bit(base, lo, lo == K), hi, hi == K);   // J up, K down
                const int c = __ldg(a.rankA + h), c2 = __ldg(a.rankA + (h ^ mask));
#pragma unroll 4
                for (int64_t r = ra; r < rb; ++r) {
                    const int64_t off = __ldg(a.row_off + __ldg(a.rows_of_m + r));
                    mul_add<T>(acc, __ldg(bra + off + c2), __ldg(ket + off + c));
                }
            }
        }
    } else {            // two B sites
        const uint32_t bJ = 1u << (J - a.nA), bK = 1u << (K - a.nA);
        for (int m = mlo; m <= mhi; ++m) {
            const int64_t ra = max(p0, a.row_base[m]), rb = min(p1, a.row_base[m + 1]);
            const int len = (int)a.ncol[m];
            for (int64_t r = ra; r < rb; ++r) {
                const int32_t row = __ldg(a.rows_of_m + r);
                const uint32_t hb = __ldg(a.row_pat + row);
                if ((hb & bJ) || !(hb & bK)) continue;
                const T *kr = ket + __ldg(a.row_off + row);
                const T *br = bra + __ldg(a.row_off + __ldg(a.rowidx + (hb ^ bJ ^ bK)));
#pragma unroll 4
                for (int c = lane; c < len; c += 32) mul_add<T>(acc, __ldg(br + c), __ldg(kr + c));
            }
        }
    }
    acc = warp_sum(acc);
    if (lane == 0) out[2 * p] = ((J + K) & 1) ? -acc : acc;
}

// Sz Sz of two B sites: with W(row) = sum over the row of b = bra ket, sum_row W s_J s_K.  A warp per
// row (one FMA per element), the row's W then goes to every pair's sum (lanes over pairs).
template <typename T>
__device__ __forceinline__ void rdm_rows(const T *__restrict__ bra, const T *__restrict__ ket, const HsRdmArgs &a,
                                         int mlo, int mhi, int chunk, double *accs, double *__restrict__ partials)
{
    // accs: [8 warps][nbb]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double *mine = accs + warp * a.nbb;
    for (int q = lane; q < a.nbb; q += 32) mine[q] = 0.0;
    const int64_t p0 = a.chunk0[chunk], p1 = a.chunk0[chunk + 1];
    for (int m = mlo; m <= mhi; ++m) {
        const int64_t ra = max(p0, a.row_base[m]), rb = min(p1, a.row_base[m + 1]);
        const int len = (int)a.ncol[m];
        for (int64_t r = ra + warp; r < rb; r += kRdmThreads / 32) {
            const int32_t row = __ldg(a.rows_of_m + r);
            const uint32_t hb = __ldg(a.row_pat + row);
            const int64_t off = __ldg(a.row_off + row);
            double w = 0.0;
#pragma unroll 4
            for (int c = lane; c < len; c += 32) w = fma((double)__ldg(bra + off + c), (double)__ldg(ket + off + c), w);
            w = warp_sum(w);
            for (int q = lane; q < a.nbb; q += 32) {
                const int p = a.bb_pair[q];
                mine[q] += (((hb >> (a.pj[p] - a.nA)) ^ (hb >> (a.pk[p] - a.nA))) & 1u) ? -w : w;
            }
        }
    }
    __syncthreads();
    for (int q = threadIdx.x; q < a.nbb; q += kRdmThreads) {
        double t = 0.0;
        for (int w = 0; w < kRdmThreads / 32; ++w) t += accs[w * a.nbb + q];
        partials[((int64_t)chunk * a.npairs + a.bb_pair[q]) * 2 + 1] = 0.25 * t;
    }
}

// The other diagonal sums: with s_j = +1 / -1 for site j+1 up / down, sum b s_J s_K is
// sum_col C(col) s_J s_K for two A sites and sum_col s_J T_K(col) for an A site J and a B site K, where
// per class m of rows C(col) = sum_row b and T_K(col) = sum_row b s_K(row) = C - 2 (sum over the rows
// with K down).  A thread owns a column; rows come in ascending pattern order, so the low half of the
// B sites costs an addition only where the bit is set (uniform over the CTA) and the high half one
// addition per run of equal high bits: about 2 + nB/4 FP64 operations per element.
constexpr int kHdThreads = kRdmThreads;

template <typename T>
__device__ __forceinline__ void rdm_diag_tile(const T *__restrict__ bra, const T *__restrict__ ket, const HsRdmArgs &a,
                                              int mlo, int mhi, int tile, double *Ts, double *__restrict__ partials)
{
    // Ts: [nB][kHdThreads], then Cs
    double *Cs = Ts + a.nB * kHdThreads;
    constexpr int LO = kMaxHalf / 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int m = mlo;
    while (m < mhi && tile >= a.tile_base[m + 1]) ++m;
    const int ncx = (int)((a.ncol[m] + kHdThreads - 1) / kHdThreads);
    const int local = tile - a.tile_base[m];
    const int cx = local % ncx, ry = local / ncx, nry = a.nry[m];
    const int64_t col = (int64_t)cx * kHdThreads + threadIdx.x;
    const bool act = col < a.ncol[m];
    const int64_t nr_m = a.row_base[m + 1] - a.row_base[m];
    const int64_t q0r = nr_m * ry / nry, q1r = nr_m * (ry + 1) / nry;
    const int nA = a.nA, lo = a.nB / 2;     // B bits [0, lo) bit by bit, [lo, nB) per run
    double C = 0.0, S = 0.0, Tl[LO], Th[LO];
#pragma unroll
    for (int k = 0; k < LO; ++k) Tl[k] = Th[k] = 0.0;
    uint32_t run = 0;
    auto flush = [&]() {
#pragma unroll
        for (int k = 0; k < LO; ++k)
            if ((run >> k) & 1u) Th[k] += S;
        C += S;
        S = 0.0;
    };
    const int32_t *rows = a.rows_of_m + a.row_base[m];
    constexpr int G = 4;                    // rows' loads in flight
    for (int64_t r0 = q0r; r0 < q1r; r0 += G) {
        double b[G];
        uint32_t hb[G];
#pragma unroll
        for (int i = 0; i < G; ++i) {
            const bool in = r0 + i < q1r;
            const int32_t row = __ldg(rows + (in ? r0 + i : q1r - 1));
            hb[i] = __ldg(a.row_pat + row);
            const int64_t at = __ldg(a.row_off + row) + col;
            b[i] = (in && act) ? (double)__ldg(bra + at) * (double)__ldg(ket + at) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < G; ++i) {
            if ((hb[i] >> lo) != run) {
                flush();
                run = hb[i] >> lo;
            }
            S += b[i];
#pragma unroll
            for (int k = 0; k < LO; ++k)
                if (k < lo && ((hb[i] >> k) & 1u)) add_branch(Tl[k], b[i]);
        }
    }
    flush();
#pragma unroll
    for (int k = 0; k < LO; ++k) {
        if (k < lo) Ts[k * kHdThreads + threadIdx.x] = C - 2.0 * Tl[k];
        if (lo + k < a.nB) Ts[(lo + k) * kHdThreads + threadIdx.x] = C - 2.0 * Th[k];
    }
    Cs[threadIdx.x] = C;
    __syncthreads();
    // sums over the tile's columns (a column past the class holds zeros): lanes over columns
    constexpr int NC = kHdThreads / 32;
    uint32_t ha[NC];
#pragma unroll
    for (int i = 0; i < NC; ++i)
        ha[i] = __ldg(a.col_pat + a.col_base[m] + min((int64_t)cx * kHdThreads + i * 32 + lane, a.ncol[m] - 1));
    for (int q = warp; q < a.npairs; q += kHdThreads / 32) {
        const int J = a.pj[q], K = a.pk[q];
        if (J >= nA && K >= nA && J != K) continue;      // rdm_rows
        const bool cross = (J < nA) != (K < nA);
        const int ja = J < nA ? J : K;
        const double *v = cross ? Ts + ((J < nA ? K : J) - nA) * kHdThreads : Cs;
        const int kA = (J == K || cross) ? 31 : K;       // bit 31 of a pattern is clear
        const int jA = (J == K) ? 31 : ja;
        double s1 = 0.0;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const double tv = v[i * 32 + lane];
            s1 += (((ha[i] >> jA) ^ (ha[i] >> kA)) & 1u) ? -tv : tv;
        }
        s1 = warp_sum(s1);
        if (lane == 0) {
            double *o = partials + ((int64_t)tile * a.npairs + q) * 2;
            if (J == K) o[0] = 0.5 * s1;
            o[1] = 0.25 * s1;
        }
    }
}

// One launch: the diagonal tiles, then the row chunks, then the flips (tasks of one chunk side by side).
template <typename T, int NB, int CTAS>
__global__ void __launch_bounds__(kRdmThreads, CTAS) heis_rdm_kernel(const T *__restrict__ bra,
                                                                     const T *__restrict__ ket,
                                                                     const __grid_constant__ HsRdmArgs a, int mlo,
                                                                     int mhi, int ntiles, int nch,
                                                                     double *__restrict__ partials)
{
    extern __shared__ __align__(16) double smem_d[];
    int b = blockIdx.x;
    if (b < ntiles) {
        rdm_diag_tile<T>(bra, ket, a, mlo, mhi, b, smem_d, partials + (int64_t)nch * 2 * a.npairs);
        return;
    }
    b -= ntiles;
    if (a.nbb > 0) {
        if (b < nch) {
            rdm_rows<T>(bra, ket, a, mlo, mhi, b, smem_d, partials);
            return;
        }
        b -= nch;
    }
    constexpr int W = kRdmThreads / 32;
    const int ng = (a.ntask + W - 1) / W;
    rdm_flips<T, NB>(bra, ket, a, mlo, mhi, (b % ng) * W + (threadIdx.x >> 5), b / ng, partials);
}

// out[p][k] = sum over the partial rows of the distinct pair of p
struct HsRdmMap {
    int16_t pair[kRdmTasks];
};

__global__ void __launch_bounds__(256) heis_rdm_reduce_kernel(const double *__restrict__ partials, int nrows, int npairs,
                                                              const __grid_constant__ HsRdmMap map, int nout,
                                                              double *__restrict__ out)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = blockIdx.x * 8 + warp;
    if (j >= 2 * nout) return;
    const int q = 2 * map.pair[j >> 1] + (j & 1);
    double s = 0.0;
    for (int b = lane; b < nrows; b += 32) s += partials[(int64_t)b * 2 * npairs + q];
    s = warp_sum(s);
    if (lane == 0) out[j] = s;
}

template <typename T>
static int heis_struct_rdm_run(ed_sector *s, cudaStream_t st, const T *bra, const T *ket, int npairs,
                               const int32_t *pairs, double *out, double *scratch, int max_blocks)
{
    const HeisStruct &h = *s->hs;
    if (h.nB > kMaxHalf) {
        set_error("B half of %d sites (at most %d)", h.nB, kMaxHalf);
        return ED_ERR_RANGE;
    }
    HsRdmArgs a;
    HsRdmMap map;     // distinct pair of each pair of the caller's list
    a.nA = h.nA;
    a.nB = h.nB;
    for (int m = 0; m <= kMaxHalf + 1; ++m) {
        a.col_base[m] = h.col_base[m];
        a.row_base[m] = h.row_base[m];
        if (m <= kMaxHalf) a.ncol[m] = h.ncol[m];
    }
    a.col_pat = h.col_pat; a.row_pat = h.row_pat;
    a.rankA = h.rankA; a.rowidx = h.rowidx; a.row_off = h.row_off;
    a.rows_of_m = h.rows_of_m;
    // distinct pairs (unordered when bra is ket) and the tasks they give
    int16_t seen[kMaxSites][kMaxSites];
    std::memset(seen, -1, sizeof(seen));
    int16_t ab_task[kMaxHalf][2];
    std::memset(ab_task, -1, sizeof(ab_task));
    a.npairs = a.nab = a.nbb = 0;
    int nother = 0;
    const bool same = (bra == ket);
    for (int p = 0; p < npairs; ++p) {
        int J = pairs[2 * p] - 1, K = pairs[2 * p + 1] - 1;
        if (same && J > K) std::swap(J, K);
        if (seen[J][K] < 0) {
            const int q = a.npairs++;
            seen[J][K] = (int16_t)q;
            a.pj[q] = (int8_t)J;
            a.pk[q] = (int8_t)K;
            const bool ja = J < h.nA, ka = K < h.nA;
            if (J != K && ja != ka) {
                const int site = ja ? J : K, bit = ja ? 0 : 1, kb = (ja ? K : J) - h.nA;   // J up: bit 0 at an A site J
                if (ab_task[site][bit] < 0) {
                    const int t = a.nab++;
                    ab_task[site][bit] = (int16_t)t;
                    a.ab_site[t] = (int8_t)site;
                    a.ab_bit[t] = (int8_t)bit;
                    a.ab_mask[t] = 0;
                }
                const int t = ab_task[site][bit];
                a.ab_mask[t] |= 1u << kb;
                a.ab_pair[t][kb] = (int16_t)q;
            } else if (J != K) {
                a.task_pair[nother++] = (int16_t)q;
                if (!ja) a.bb_pair[a.nbb++] = (int16_t)q;
            }
        }
        map.pair[p] = seen[J][K];
    }
    a.ntask = a.nab + nother;
    // diagonal tiles: per class m, 256-column tiles times row ranges, about one per SM (a tile's sums over
    // the pairs cost more than its rows)
    const int64_t dim = s->dim;
    const int want_tiles = std::min(num_sms(), max_blocks);
    int ntiles = 0;
    for (int m = 0; m <= kMaxHalf + 1; ++m) a.tile_base[m] = 0;
    for (int m = h.mlo; m <= h.mhi; ++m) {
        a.tile_base[m] = ntiles;
        const int64_t nr_m = h.row_base[m + 1] - h.row_base[m];
        const int ncx = (int)((h.ncol[m] + kHdThreads - 1) / kHdThreads);
        const double share = dim > 0 ? (double)(h.ncol[m] * nr_m) / (double)dim : 0.0;
        int nry = (int)std::max<double>(1.0, std::floor(share * want_tiles / std::max(ncx, 1)));
        nry = (int)std::min<int64_t>(std::max<int64_t>(nr_m, 1), nry);
        a.nry[m] = nry;
        ntiles += ncx * nry;
    }
    a.tile_base[h.mhi + 1] = ntiles;
    // row chunks: rows [0, nrows) of rows_of_m, cut where the states before them pass i/nch of all
    const bool large = dim >= kRdmLarge;
    const int nch = (int)std::max<int64_t>(1, std::min<int64_t>({h.nrows, kRdmChunks, 3 * max_blocks - ntiles}));
    if (nch + ntiles > 3 * max_blocks) {
        set_error("spin-correlation pass needs %d partial rows (scratch holds %d)", nch + ntiles, 3 * max_blocks);
        return ED_ERR_RANGE;
    }
    {
        int m = h.mlo;
        int64_t before = 0;     // states of the classes below m
        for (int i = 0; i <= nch; ++i) {
            const int64_t want = (int64_t)((double)dim * i / nch);
            while (m < h.mhi && before + h.ncol[m] * (h.row_base[m + 1] - h.row_base[m]) <= want) {
                before += h.ncol[m] * (h.row_base[m + 1] - h.row_base[m]);
                ++m;
            }
            const int64_t r = h.row_base[m] + (want - before) / std::max<int64_t>(h.ncol[m], 1);
            a.chunk0[i] = (int)std::min<int64_t>(i == nch ? h.nrows : r, h.nrows);
        }
        a.chunk0[0] = 0;
    }
    // partial rows [0, nch): flips and two-B-site sums of each chunk; [nch, nch + ntiles): the tiles
    ED_CHECK_CUDA(cudaMemsetAsync(scratch, 0, sizeof(double) * 2 * (size_t)a.npairs * (nch + ntiles), st));
    constexpr int W = kRdmThreads / 32;
    const size_t smem = sizeof(double) * std::max((size_t)(h.nB + 1) * kHdThreads, (size_t)W * a.nbb);
    auto *kfn = h.nB > 12 ? heis_rdm_kernel<T, kMaxHalf, 5>
                : large   ? heis_rdm_kernel<T, 12, 5>
                : h.nB > 8 ? heis_rdm_kernel<T, 12, 3> : heis_rdm_kernel<T, 8, 3>;
    if (smem > 48 * 1024)
        ED_CHECK_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int nblk = ntiles + (a.nbb > 0 ? nch : 0) + (a.ntask + W - 1) / W * nch;
    kfn<<<nblk, kRdmThreads, smem, st>>>(bra, ket, a, h.mlo, h.mhi, ntiles, nch, scratch);
    ED_CHECK_LAUNCH();
    heis_rdm_reduce_kernel<<<(2 * npairs + 7) / 8, 256, 0, st>>>(scratch, nch + ntiles, a.npairs, map, npairs, out);
    ED_CHECK_LAUNCH();
    return ED_OK;
}

int heis_struct_rdm(ed_sector *s, cudaStream_t st, int dtype, const void *bra, const void *ket, int npairs,
                    const int32_t *pairs, double *out, double *scratch, int max_blocks)
{
    if (!s->hs) {
        set_error("Heisenberg sector without its row tables");
        return ED_ERR_ARG;
    }
    if (dtype == ED_F32)
        return heis_struct_rdm_run<float>(s, st, static_cast<const float *>(bra), static_cast<const float *>(ket),
                                          npairs, pairs, out, scratch, max_blocks);
    return heis_struct_rdm_run<double>(s, st, static_cast<const double *>(bra), static_cast<const double *>(ket),
                                       npairs, pairs, out, scratch, max_blocks);
}

template <typename T>
static int heis_struct_run(ed_sector *s, cudaStream_t st, const T *x, T *y, double scale, double *dots,
                           double *partials)
{
    const HeisStruct &h = *s->hs;
    HsArgs a;
    a.nA = h.nA;
    a.nB = h.nB;
    a.nab = h.nab;
    a.nrows = h.nrows;
    for (int m = 0; m <= kMaxHalf + 1; ++m) {
        a.col_base[m] = h.col_base[m];
        a.slice_base[m] = h.slice_base[m];
        a.row_base[m] = h.row_base[m];
        if (m <= kMaxHalf) a.ncol[m] = h.ncol[m];
    }
    a.col_pat = h.col_pat; a.row_pat = h.row_pat;
    a.rankA = h.rankA; a.aa_off = (sizeof(T) == 4) ? h.aa_off : h.aa64_off; a.aa64_src = h.aa64_src; a.aa64_col = h.aa64_col; a.row_m = h.row_m;
    a.rowidx = h.rowidx; a.bb_ptr = h.bb_ptr; a.bb_src = h.bb_src; a.rows_of_m = h.rows_of_m;
    a.row_off = h.row_off;
    a.diagA = (sizeof(T) == 4) ? (const void *)h.diagA32 : (const void *)h.diagA;
    a.diagB = (sizeof(T) == 4) ? (const void *)h.diagB32 : (const void *)h.diagB;
    a.aa64_cf = h.aa64_cf;
    a.aa_pk32 = h.aa_pk32;
    a.col_abbits = h.col_abbits;
    a.row_bbits = h.row_bbits;
    a.ab_rank = h.ab_rank;
    a.ab_lut = (sizeof(T) == 4) ? (const void *)h.ab_lut32 : (const void *)h.ab_lut;
    a.ncols = h.ncols;
    a.ab_fast = h.ab_fast ? 1 : 0;
    a.bb_cf = (sizeof(T) == 4) ? (const void *)h.bb_cf32 : (const void *)h.bb_cf64;
    for (int q = 0; q < h.nab; ++q) {
        a.ab_pa[q] = h.ab_pa[q]; a.ab_pb[q] = h.ab_pb[q];
        a.ab_fjk[q] = h.ab_fjk[q]; a.ab_fkj[q] = h.ab_fkj[q]; a.ab_zz[q] = h.ab_zz[q];
    }
    a.scale = scale;
    for (int m = 0; m <= h.nA; ++m) a.m_order[m] = (int8_t)m;
    std::sort(a.m_order, a.m_order + h.nA + 1, [&](int8_t x, int8_t y) { return h.ncol[x] > h.ncol[y]; });
    const int nsm = num_sms();
    // rows by length give the CTAs even shares (FP64: 4x6 157 -> 149 us, 4x7 3.69 -> 3.51 ms; FP32 here only
    // with more than 32 A-B bonds: all couplings, 24 sites 570 -> 541 us, 26 2.40 -> 2.30 ms, but 22 148 -> 163);
    // vectors far above L2 keep memory order, where the A-B bonds' source rows are near (4x8: 60 ms, by length
    // 67; on a ring with next-but-three neighbours the two are level: 30 sites 14.6 and 14.0), and so do rows
    // that have a CTA each (4x4: the row pass 5.5 us, by length 6.6: the look-up leads the chain of loads)
    a.by_length = (double)s->dim * sizeof(T) <= kL2Bytes && h.nrows > (int64_t)nsm * 4 ? 1 : 0;
    // ---- pass R
    const int maxsm = max_smem();
    const size_t smem4 = heis_col4_head_bytes(h.nab) + (size_t)std::max<int64_t>(h.max_len, 1) * 16;
    // FP32 with the packed A-B path: four rows of one hole count per CTA when their columns
    // fit (PYHUB_ED_HEIS_ROWS=1 selects the one-row pass; both give the same product)
    const char *one = std::getenv("PYHUB_ED_HEIS_ROWS");
    if (sizeof(T) == 4 && h.ab_fast && smem4 <= (size_t)maxsm && !(one && one[0] == '1')) {
        int64_t nitems = 0;
        for (int m = 0; m <= h.nA; ++m) nitems += (h.row_base[m + 1] - h.row_base[m] + 3) / 4;
        if (smem4 > 48 * 1024)
            ED_CHECK_CUDA(cudaFuncSetAttribute(heis_row_col4_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)smem4));
        // two CTAs of 512 threads per SM where two groups of rows fit (one stages while the other works)
        const int threads = 2 * (smem4 + 1024) <= (size_t)maxsm ? 512 : kHeisCol4Threads;
        int64_t blocks = std::min<int64_t>(nitems, (int64_t)nsm * (threads == 512 ? 2 : 1));
        if (blocks < 1) blocks = 1;
        heis_row_col4_kernel<<<(unsigned)blocks, threads, smem4, st>>>(
            reinterpret_cast<const float *>(x), reinterpret_cast<float *>(y), a, nitems);
    } else {
        const size_t smem = heis_row_head_bytes(h.nab, sizeof(T)) + (size_t)std::max<int64_t>(h.max_len, 1) * sizeof(T);
        if (smem > 48 * 1024)
            ED_CHECK_CUDA(cudaFuncSetAttribute(heis_row_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int64_t blocks = std::min<int64_t>(h.nrows, (int64_t)nsm * 4);
        if (blocks < 1) blocks = 1;
        heis_row_kernel<T><<<(unsigned)blocks, kHeisRowThreads, smem, st>>>(x, y, a);
    }
    ED_CHECK_LAUNCH();
    // ---- pass S: one wave of resident CTAs walks the items (slab, eight rows).  A slab takes at most
    // 20 MB of L2 in FP32 (48 / 30 / 20 / 10 MB: 4x7 864 / 821 / 811 / 828 us, 5x6 3.71 / 3.65 / 3.29 / 3.36
    // ms, 4x8 15.3 / 15.5 / 13.5-14.2 / 13.5), 48 MB in FP64 (4x7 3.20 against 3.22 ms, 4x8 55.9 against 56.8,
    // 5x6 15.1 against 14.9); small sectors cut the columns further, down to one pass of 128, until every CTA
    // has several items (a share of 3.4 items each would leave a wave 15% empty).
    const double slab_bytes = sizeof(T) == 4 ? 20.0e6 : 48.0e6;
    SlabPlan p;
    p.nblk = 0;
    p.item_base[0] = 0;
    int64_t blocks2 = std::min<int64_t>((int64_t)nsm * kHeisSlabCtas, kMaxPartialBlocksHeis);
    int64_t groups = 0;
    for (int m = 0; m <= h.nA; ++m) groups += (h.row_base[m + 1] - h.row_base[m] + 7) / 8;
    const int64_t cuts = std::max<int64_t>(1, 8 * blocks2 / std::max<int64_t>(groups, 1));
    for (int m = 0; m <= h.nA; ++m) {
        const int64_t nr = h.row_base[m + 1] - h.row_base[m];
        if (nr == 0) continue;
        const int64_t len = h.ncol[m];
        int64_t w = (int64_t)(slab_bytes / ((double)nr * sizeof(T)));
        w = w / 32 * 32;
        if (w < 256) w = 256;
        w = std::min(w, std::max<int64_t>(128, (len / cuts + 127) / 128 * 128));
        if (w > len) w = len;
        const int b = p.nblk++;
        p.m[b] = m;
        p.slab_w[b] = w;
        p.ngroups[b] = (nr + 7) / 8;
        p.item_base[b + 1] = p.item_base[b] + ((len + w - 1) / w) * p.ngroups[b];
    }
    if (blocks2 > p.item_base[p.nblk]) blocks2 = p.item_base[p.nblk];
    if (blocks2 < 1) blocks2 = 1;
    heis_slab_kernel<T><<<(unsigned)blocks2, 256, 0, st>>>(x, y, a, p, dots ? partials : nullptr);
    ED_CHECK_LAUNCH();
    if (dots) return launch_reduce(partials, (int)blocks2, 2, dots, st);
    return ED_OK;
}

int heis_struct_hv(ed_sector *s, cudaStream_t st, int dtype, const void *x, void *y, double scale, double *dots,
                   double *partials)
{
    if (!s->hs) {
        set_error("Heisenberg sector without its row tables");
        return ED_ERR_ARG;
    }
    if (dtype == ED_F32)
        return heis_struct_run<float>(s, st, static_cast<const float *>(x), static_cast<float *>(y), scale, dots,
                                      partials);
    return heis_struct_run<double>(s, st, static_cast<const double *>(x), static_cast<double *>(y), scale, dots,
                                   partials);
}

}  // namespace ed
