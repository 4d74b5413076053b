// Export of a block matrix (K or M) in the reference's layout: CSC over the equation numbers, the scalar entries that
// the keep bits mark, rows ascending in each column (src/mech/mech-solver.jl:78-110 builds it with sparse()).
//
// The columns are made on the device, a warp per column, and read back in chunks of a bounded workspace: per column a
// walk over the node's block row, whose pattern is symmetric, so that the blocks of the column are the transposed
// positions.  On the host the same walk, the scatter and a sort per column took 9 ms for 1.27 million entries (29 x 13 x
// 13 HEX8); the count now takes 0.04 ms and the export 0.25 ms, of which the read-back of 20 MB is most.
// Few entries are still walked on the host, where the launches and their arrays cost more: both calls that a mount takes
// (the count, then all) 43 us instead of 107 for 576 entries, 85 instead of 117 for 7 200; 117 and 119 for 11 700, 136
// and 118 for 15 800.
#include "amr_internal.h"

#include <algorithm>

namespace {

constexpr size_t kCscChunk = size_t(1) << 21;  // entries of a chunk, 32 bytes each: 64 MB at most
constexpr size_t kCscMin = size_t(1) << 15;    // below this a failed allocation is an error
constexpr int64_t kCscHost = 12000;            // entries of the blocks up to which the host makes the columns

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

__global__ void k_csc_slot(int64_t nnodes, const int64_t *eq_id, int64_t *slot) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 3 * nnodes) return;
    const int64_t e = eq_id[t];
    if (e >= 0) slot[e] = t;
}

// position of column j in block row [a, b) (ascending columns); the pattern is symmetric, so it is there
__device__ __forceinline__ int64_t find_block(const int32_t *bcol, int64_t a, int64_t b, int32_t j) {
    while (a < b) {
        const int64_t mid = (a + b) >> 1;
        if (bcol[mid] < j) a = mid + 1;
        else b = mid;
    }
    return a;
}

// FILL false: the entries of each column.  FILL true: columns [c0, c1), whose entries go to [colptr[col] - colptr[c0]):
// first in the order of the nodes (ur, us), then each at the number of smaller rows in its column.
template <int B, bool FILL>
__global__ void __launch_bounds__(256)
    k_csc_column(int64_t c0, int64_t c1, const int64_t *slot, const int64_t *brow_ptr, const int32_t *bcol,
                 const int64_t *eq_id, const uint16_t *keep, const double *vals, int64_t bstride, int32_t *cnt,
                 const int64_t *colptr, int64_t *ur, int64_t *us, int64_t *rowval, double *nzval) {
    const int64_t col = c0 + ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x & 31;
    if (col >= c1) return;
    const int32_t j = (int32_t)(slot[col] / 3);
    const int d = (int)(slot[col] % 3);
    const int64_t k0 = brow_ptr[j], k1 = brow_ptr[j + 1];
    const int64_t base = FILL ? colptr[col] - colptr[c0] : 0;
    int64_t n = 0;  // entries so far
    for (int64_t kb = k0; kb < k1; kb += 32) {
        unsigned bits = 0;  // kept rows of this lane's block in column d
        int64_t k = 0;
        int32_t node = 0;
        if (kb + lane < k1) {
            node = bcol[kb + lane];
            const int64_t a = brow_ptr[node], b = brow_ptr[node + 1];
            k = find_block(bcol, a, b, j);
            if (k < b && bcol[k] == j)
                for (int c = 0; c < B; c++)
                    if ((keep[k] >> (c * B + d) & 1) && eq_id[3 * (int64_t)node + c] >= 0) bits |= 1u << c;
        }
        const int mine = __popc(bits);
        int incl = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (FILL) {
            int64_t p = base + n + incl - mine;
            for (int c = 0; c < B; c++)
                if (bits >> c & 1) {
                    ur[p] = eq_id[3 * (int64_t)node + c];
                    us[p] = (int64_t)(c * B + d) * bstride + k;
                    p++;
                }
        }
        n += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (!FILL) {
        if (lane == 0) cnt[col] = (int32_t)n;
        return;
    }
    __syncwarp();
    for (int64_t p = 0; p < n; p += 32) {  // rows are distinct: a rank is a place
        const bool in = p + lane < n;
        const int64_t r = in ? ur[base + p + lane] : 0;
        int64_t rank = 0;
        for (int64_t q = 0; q < n; q++) rank += ur[base + q] < r;
        if (in) {
            rowval[base + rank] = r;
            if (nzval) nzval[base + rank] = vals[us[base + p + lane]];
        }
    }
}

// the device arrays of one export
struct CscScratch {
    int64_t *slot = nullptr, *colptr = nullptr, *ur = nullptr, *us = nullptr, *rv = nullptr;
    int32_t *cnt = nullptr;
    double *nz = nullptr;
    void free_chunk() {
        amr_free(ur); amr_free(us); amr_free(rv); amr_free(nz);
    }
    ~CscScratch() {
        amr_free(slot); amr_free(colptr); amr_free(cnt);
        free_chunk();
    }
};

template <int B, bool FILL>
void columns(amr_model *m, const CscScratch &w, int64_t c0, int64_t c1, const uint16_t *keep, const double *vals,
             bool nz) {
    k_csc_column<B, FILL><<<nblk(c1 - c0, 8), 256, 0, m->stream>>>(c0, c1, w.slot, m->brow_ptr, m->bcol, m->eq_id, keep,
                                                                   vals, m->bstride, w.cnt, w.colptr, w.ur, w.us, w.rv,
                                                                   nz ? w.nz : nullptr);
    AMR_COUNT(1);
    AMR_CUDA(cudaGetLastError());
}

// the same on the host: entries by walking the rows, then each column sorted by its rows
void host_csc(amr_model *m, int64_t *nnz_out, int64_t *colptr, int64_t *rowval, double *nzval, const uint16_t *d_keep,
              const double *d_vals) {
    const int B = m->B;
    std::vector<uint16_t> keep(m->nblocks);
    std::vector<double> vals;
    amr_d2h(m, keep.data(), d_keep, m->nblocks * sizeof(uint16_t));
    if (colptr && nzval) {
        vals.resize((size_t)m->bstride * m->BB);
        amr_d2h(m, vals.data(), d_vals, vals.size() * sizeof(double));
    }
    const std::vector<int64_t> &eq = m->h_eq_id;
    auto walk = [&](auto entry) {
        for (int64_t n = 0; n < m->nnodes; n++)
            for (int64_t k = m->h_brow_ptr[n]; k < m->h_brow_ptr[n + 1]; k++)
                for (int q = 0; q < m->BB; q++) {
                    const int64_t r = eq[3 * n + q / B], c = eq[3 * (int64_t)m->h_bcol[k] + q % B];
                    if (r >= 0 && c >= 0 && (keep[k] >> q & 1)) entry(r, c, (size_t)q * m->bstride + k);
                }
    };
    std::vector<int64_t> at(m->ndofs + 1, 0);
    walk([&](int64_t, int64_t c, size_t) { at[c + 1]++; });
    for (int64_t i = 0; i < m->ndofs; i++) at[i + 1] += at[i];
    *nnz_out = at[m->ndofs];
    if (!colptr) return;
    std::copy(at.begin(), at.end(), colptr);
    std::vector<std::pair<int64_t, size_t>> e(*nnz_out);  // row, place of the value
    walk([&](int64_t r, int64_t c, size_t v) { e[at[c]++] = {r, v}; });
    for (int64_t c = 0; c < m->ndofs; c++) std::sort(e.begin() + colptr[c], e.begin() + colptr[c + 1]);
    for (int64_t i = 0; i < *nnz_out; i++) {
        rowval[i] = e[i].first;
        if (nzval) nzval[i] = vals[e[i].second];
    }
}

}  // namespace

void amr_export_csc(amr_model *m, int64_t *nnz_out, int64_t *colptr, int64_t *rowval, double *nzval, const uint16_t *keep,
                    const double *vals) {
    const int64_t nd = m->ndofs;
    *nnz_out = 0;
    if (nd == 0) {
        if (colptr) colptr[0] = 0;
        return;
    }
    if (m->nblocks * m->BB <= kCscHost) {
        host_csc(m, nnz_out, colptr, rowval, nzval, keep, vals);
        return;
    }
    CscScratch w;
    amr_alloc(&w.slot, nd);
    amr_alloc(&w.cnt, nd);
    k_csc_slot<<<nblk(3 * m->nnodes, 256), 256, 0, m->stream>>>(m->nnodes, m->eq_id, w.slot);
    AMR_COUNT(1);
    AMR_CUDA(cudaGetLastError());
    if (m->B == 3) columns<3, false>(m, w, 0, nd, keep, vals, false);
    else columns<2, false>(m, w, 0, nd, keep, vals, false);
    std::vector<int32_t> cnt(nd);
    amr_d2h(m, cnt.data(), w.cnt, nd * sizeof(int32_t));
    if (!colptr) {
        int64_t s = 0;
        for (int64_t i = 0; i < nd; i++) s += cnt[i];
        *nnz_out = s;
        return;
    }
    int64_t most = 1;
    colptr[0] = 0;
    for (int64_t i = 0; i < nd; i++) {
        colptr[i + 1] = colptr[i] + cnt[i];
        most = std::max<int64_t>(most, cnt[i]);
    }
    *nnz_out = colptr[nd];
    if (colptr[nd] == 0) return;
    amr_alloc(&w.colptr, nd + 1);
    amr_h2d(m, w.colptr, colptr, (nd + 1) * sizeof(int64_t));
    int64_t cap = std::max<int64_t>(most, std::min<int64_t>(colptr[nd], kCscChunk));
    for (;;) {
        try {
            amr_alloc(&w.ur, cap);
            amr_alloc(&w.us, cap);
            amr_alloc(&w.rv, cap);
            if (nzval) amr_alloc(&w.nz, cap);
            break;
        } catch (const AmrError &e) {
            w.free_chunk();
            if (e.code != AMR_ENOMEM || cap <= std::max<int64_t>(most, kCscMin)) throw;
            cap = std::max<int64_t>(most, cap / 2);
        }
    }
    for (int64_t c0 = 0; c0 < nd;) {
        const int64_t c1 = std::upper_bound(colptr + c0 + 1, colptr + nd + 1, colptr[c0] + cap) - colptr - 1;
        const int64_t n = colptr[c1] - colptr[c0];
        if (m->B == 3) columns<3, true>(m, w, c0, c1, keep, vals, nzval != nullptr);
        else columns<2, true>(m, w, c0, c1, keep, vals, nzval != nullptr);
        amr_d2h(m, rowval + colptr[c0], w.rv, n * sizeof(int64_t));
        if (nzval) amr_d2h(m, nzval + colptr[c0], w.nz, n * sizeof(double));
        c0 = c1;
    }
}
