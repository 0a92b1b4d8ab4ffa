// Masked SpGEMM C<M> = A (+.x) B by sorted-list intersection.
//
// Replaces SpMSpM_masked_ikj (src/backend/spmspm/spmspm_masked_hash_based_gustavson.h:9-168),
// which builds a hash set per mask row and a hash map of partial sums.  On
// the GPU every stored (i, j) of the mask is one intersection of row i of A
// with column j of B (both sorted): a warp takes 32 consecutive mask
// entries and, entry by entry, its lanes split the shorter list and binary
// search each element in the longer one, so a hub pair is spread over the
// warp and light pairs cost a few instructions each.
//
// Unmasked SpGEMM C = A (+.x) B replaces SpMSpM_unmasked_ikj
// (src/backend/spmspm/spmspm_hash_based_gustavson.h:9-148, a hash map per
// row of C) by sums in column windows (spgemm_window.cu) and, for the operands
// those refuse, by expand-sort-compress in row blocks: every product
// A_ik * B_kj is written with its (i, j) key (one thread per product, found
// by binary search over the per-entry product offsets), the block is radix
// sorted by key, equal keys are reduced with the semiring's add, and sums
// equal to 0 are dropped as the reference keeps only val != 0.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstdlib>
#include <vector>

#include "common.cuh"
#include "internal.h"

namespace gbk {

namespace {

template <int SR, typename C, typename AT>
__global__ void k_masked_spgemm(const int32_t* __restrict__ mptr, const int32_t* __restrict__ midx, int64_t mrows,
                                int64_t mnnz, const int32_t* __restrict__ aptr, const int32_t* __restrict__ aidx,
                                const AT* __restrict__ aval, const int32_t* __restrict__ bptr,
                                const int32_t* __restrict__ bidx, const AT* __restrict__ bval, C* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t groups = (mnnz + 31) / 32;
    for (int64_t g = warp; g < groups; g += nwarps) {
        const int64_t e0 = g * 32;
        // row of the first entry of this group; later entries advance from it
        int64_t lo = 0, hi = mrows;
        while (hi - lo > 1) {
            int64_t mid = (lo + hi) >> 1;
            if (mptr[mid] <= e0)
                lo = mid;
            else
                hi = mid;
        }
        int64_t row = lo;
        const int64_t e_end = min(e0 + 32, mnnz);
        C my_out = C(0);
        for (int64_t e = e0; e < e_end; e++) {
            while (mptr[row + 1] <= e) row++;
            const int32_t j = midx[e];
            int32_t a0 = aptr[row], a1 = aptr[row + 1];
            int32_t b0 = bptr[j], b1 = bptr[j + 1];
            // lanes walk the shorter list, binary-search the longer
            const bool a_short = (a1 - a0) <= (b1 - b0);
            const int32_t s0 = a_short ? a0 : b0, s1 = a_short ? a1 : b1;
            const int32_t l0 = a_short ? b0 : a0, l1 = a_short ? b1 : a1;
            const int32_t* sidx = a_short ? aidx : bidx;
            const int32_t* lidx = a_short ? bidx : aidx;
            C acc = C(0);
            for (int32_t p = s0 + lane; p < s1; p += 32) {
                const int32_t key = sidx[p];
                int32_t lo2 = l0, hi2 = l1;
                while (lo2 < hi2) {
                    int32_t mid = (lo2 + hi2) >> 1;
                    if (lidx[mid] < key)
                        lo2 = mid + 1;
                    else
                        hi2 = mid;
                }
                if (lo2 < l1 && lidx[lo2] == key) {
                    if (SR == GBK_PLUS_ONE) {
                        acc += C(1);
                    } else {
                        const int32_t pa = a_short ? p : lo2;
                        const int32_t pb = a_short ? lo2 : p;
                        acc += C(aval[pa]) * C(bval[pb]);
                    }
                }
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
            const C total = __shfl_sync(0xffffffffu, acc, 0);
            if (lane == (int)(e - e0)) my_out = total;
        }
        if (e0 + lane < e_end) out[e0 + lane] = my_out;
    }
}

// ---------------------------------------------------------------------------
// unmasked SpGEMM

// products of A's entry e: the degree of row aidx[e] of B
__global__ void k_entry_products(const int32_t* __restrict__ aidx, int64_t nnz, const int32_t* __restrict__ bptr,
                                 int64_t* __restrict__ cnt) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < nnz) cnt[e] = bptr[aidx[e] + 1] - bptr[aidx[e]];
}

// product offset of each row's first entry
__global__ void k_row_offsets(const int32_t* __restrict__ aptr, int64_t nrows, const int64_t* __restrict__ off,
                              int64_t* __restrict__ roff) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r <= nrows) roff[r] = off[aptr[r]];
}

// row of A's entry e
__global__ void k_entry_rows(const int32_t* __restrict__ aptr, int64_t nrows, int64_t nnz, int32_t* __restrict__ arow) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nnz) return;
    int64_t lo = 0, hi = nrows;  // last row starting at or before e
    while (hi - lo > 1) {
        const int64_t mid = (lo + hi) >> 1;
        if (aptr[mid] <= e)
            lo = mid;
        else
            hi = mid;
    }
    arow[e] = (int32_t)lo;
}

// Products [p0, p1) of the entries [e0, e1) (off: exclusive product offsets
// per entry, off[e1] = p1): key ((row - row0) << colbits | column), value
// mul(a, b); the short keys keep the radix sort to the bits in use.
template <int SR, typename T>
__global__ void k_expand(const int64_t* __restrict__ off, int64_t e0, int64_t e1, int64_t p0, int64_t p1,
                         const int32_t* __restrict__ arow, int32_t row0, int colbits, const int32_t* __restrict__ aidx,
                         const T* __restrict__ aval,
                         const int32_t* __restrict__ bptr, const int32_t* __restrict__ bidx,
                         const T* __restrict__ bval, unsigned long long* __restrict__ key, T* __restrict__ val) {
    using S = Semiring<SR, T>;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = p0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < p1; p += stride) {
        int64_t lo = e0, hi = e1;  // last entry whose products start at or before p
        while (hi - lo > 1) {
            const int64_t mid = (lo + hi) >> 1;
            if (off[mid] <= p)
                lo = mid;
            else
                hi = mid;
        }
        const int32_t k = aidx[lo];
        const int64_t f = bptr[k] + (p - off[lo]);
        key[p - p0] = ((unsigned long long)(uint32_t)(arow[lo] - row0) << colbits) | (unsigned long long)(uint32_t)bidx[f];
        val[p - p0] = S::mul(aval[lo], bval[f]);
    }
}

template <int SR, typename T>
struct SemiringAdd {
    __device__ __forceinline__ T operator()(const T& a, const T& b) const { return Semiring<SR, T>::add(a, b); }
};

template <typename T>
struct NonZero {
    __device__ __forceinline__ bool operator()(const T& v) const { return v != T(0); }
};

__global__ void k_split_keys(const unsigned long long* __restrict__ key, int64_t n, int32_t row0, int colbits,
                             int32_t* __restrict__ row, int32_t* __restrict__ col) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    row[i] = row0 + (int32_t)(key[i] >> colbits);
    col[i] = (int32_t)(key[i] & ((1ull << colbits) - 1));
}

// ptr[r] = first entry of row >= r (rows ascending)
__global__ void k_bounds(const int32_t* __restrict__ row, int64_t nnz, int64_t nrows, int32_t* __restrict__ ptr) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i > nnz) return;
    const int64_t lo = i == 0 ? 0 : (int64_t)row[i - 1] + 1;
    const int64_t hi = i == nnz ? nrows : (int64_t)row[i];
    for (int64_t r = lo; r <= hi; ++r) ptr[r] = (int32_t)i;
}

template <typename T>
__global__ void k_nonzero_flags(const T* __restrict__ v, int64_t n, uint8_t* __restrict__ flag) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) flag[i] = v[i] != T(0);
}

unsigned nb(int64_t n) { return (unsigned)std::max<int64_t>(1, (n + 255) / 256); }

// Products per block: keys, values and their sorted copies, about 24 bytes
// each.  GBK_MXM_BLOCK_PRODUCTS (at least 1) overrides it, so small products
// can exercise several blocks.
constexpr int64_t kBlockProductsDefault = 64ll << 20;

int64_t block_products() {
    const char* e = getenv("GBK_MXM_BLOCK_PRODUCTS");
    const long long v = e ? atoll(e) : 0;
    return v >= 1 ? (int64_t)v : kBlockProductsDefault;
}

template <int SR, typename T>
int mxm_unmasked(gbk_matrix* out, const CsrView& a, const CsrView& b, cudaStream_t s) {
    const int64_t n = a.nrows, m = b.ncols, annz = a.nnz;
    StreamScratch dev(s);
    auto need = [&](int rc) { return rc == GBK_SUCCESS; };
    int64_t* off = nullptr;
    int32_t* arow = nullptr;
    if (!need(dev.get(&off, 8 * (annz + 1))) || !need(dev.get(&arow, 4 * annz))) {
        set_error("gbk_mxm: out of device memory");
        return GBK_OUT_OF_MEMORY;
    }
    if (annz > 0) {
        k_entry_products<<<nb(annz), 256, 0, s>>>(a.idx, annz, b.ptr, off);
        GBK_LAUNCHED();
        k_entry_rows<<<nb(annz), 256, 0, s>>>(a.ptr, n, annz, arow);
        GBK_LAUNCHED();
    }
    GBK_CUDA(cudaMemsetAsync(off + annz, 0, 8, s));
    {
        size_t tb = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, tb, off, off, annz + 1, s);
        void* tmp = nullptr;
        if (!need(dev.get(&tmp, tb))) return GBK_OUT_OF_MEMORY;
        GBK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, off, off, annz + 1, s));
        count_launch(1);
    }
    // product offsets at row starts, on the host, to cut row blocks
    int64_t* roff = nullptr;
    if (!need(dev.get(&roff, 8 * (n + 1)))) return GBK_OUT_OF_MEMORY;
    k_row_offsets<<<nb(n + 1), 256, 0, s>>>(a.ptr, n, off, roff);
    GBK_LAUNCHED();
    std::vector<int32_t> hptr(n + 1);
    std::vector<int64_t> hroff(n + 1);
    GBK_CUDA(cudaMemcpyAsync(hptr.data(), a.ptr, 4 * (n + 1), cudaMemcpyDeviceToHost, s));
    GBK_CUDA(cudaMemcpyAsync(hroff.data(), roff, 8 * (n + 1), cudaMemcpyDeviceToHost, s));
    GBK_CUDA(cudaStreamSynchronize(s));
    // blocks of whole rows with at most kBlockProducts products (a single row may exceed it)
    std::vector<int64_t> cuts{0};
    const int64_t kBlockProducts = block_products();
    {
        int64_t r = 0;
        while (r < n) {
            const int64_t base = hroff[r];
            int64_t r1 = r + 1;
            int64_t lo = r + 1, hi = n;  // furthest row end within the budget
            while (lo <= hi) {
                const int64_t mid = (lo + hi) / 2;
                if (hroff[mid] - base <= kBlockProducts) {
                    r1 = mid;
                    lo = mid + 1;
                } else {
                    hi = mid - 1;
                }
            }
            cuts.push_back(r1);
            r = r1;
        }
    }
    int64_t maxp = 0;
    for (size_t c = 0; c + 1 < cuts.size(); ++c)
        maxp = std::max<int64_t>(maxp, hroff[cuts[c + 1]] - hroff[cuts[c]]);
    unsigned long long *key = nullptr, *key2 = nullptr;
    T *val = nullptr, *val2 = nullptr;
    int64_t* nsel = nullptr;
    if (!need(dev.get(&key, 8 * maxp)) || !need(dev.get(&key2, 8 * maxp)) || !need(dev.get(&val, sizeof(T) * maxp)) ||
        !need(dev.get(&val2, sizeof(T) * maxp)) || !need(dev.get(&nsel, 16))) {
        set_error("gbk_mxm: out of device memory for %lld products per block", (long long)maxp);
        return GBK_OUT_OF_MEMORY;
    }
    // scratch sized for the largest block
    size_t t_sort = 0, t_red = 0, t_sel = 0;
    int rowbits = 1;
    while ((1ll << rowbits) < n) ++rowbits;
    int colbits = 1;
    while ((1ll << colbits) < m) ++colbits;
    cub::DeviceRadixSort::SortPairs(nullptr, t_sort, key, key2, val, val2, maxp, 0, rowbits + colbits, s);
    cub::DeviceReduce::ReduceByKey(nullptr, t_red, key2, key, val2, val, nsel, SemiringAdd<SR, T>(), maxp, s);
    uint8_t* flag = nullptr;
    if (!need(dev.get(&flag, maxp))) return GBK_OUT_OF_MEMORY;
    cub::DeviceSelect::Flagged(nullptr, t_sel, key, flag, key2, nsel + 1, maxp, s);
    size_t t_if = 0;
    cub::DeviceSelect::If(nullptr, t_if, val, val2, nsel, maxp, NonZero<T>(), s);
    void* tmp = nullptr;
    const size_t tbytes = std::max(std::max(t_sort, t_red), std::max(t_sel, t_if)) + 256;
    if (!need(dev.get(&tmp, tbytes))) return GBK_OUT_OF_MEMORY;
    // per block: expand, sort, reduce, drop zeros; the kept entries are appended
    std::vector<unsigned long long*> okeys;
    std::vector<T*> ovals;
    std::vector<int64_t> ocnt;
    std::vector<int64_t> orow0;  // first row of each kept block
    int64_t total = 0;
    for (size_t c = 0; c + 1 < cuts.size(); ++c) {
        const int64_t e0 = hptr[cuts[c]], e1 = hptr[cuts[c + 1]];
        const int64_t p0 = hroff[cuts[c]], p1 = hroff[cuts[c + 1]], np = p1 - p0;
        if (np == 0) continue;
        const unsigned grid = (unsigned)std::min<int64_t>(nb(np), (int64_t)num_sms() * 32);
        k_expand<SR, T><<<grid, 256, 0, s>>>(off, e0, e1, p0, p1, arow, (int32_t)cuts[c], colbits, a.idx,
                                             (const T*)a.val, b.ptr, b.idx, (const T*)b.val, key, val);
        GBK_LAUNCHED();
        int brows = 1;  // bits of the block's row span
        while ((1ll << brows) < cuts[c + 1] - cuts[c]) ++brows;
        size_t tb = tbytes;
        GBK_CUDA(cub::DeviceRadixSort::SortPairs(tmp, tb, key, key2, val, val2, np, 0, brows + colbits, s));
        tb = tbytes;
        GBK_CUDA(cub::DeviceReduce::ReduceByKey(tmp, tb, key2, key, val2, val, nsel, SemiringAdd<SR, T>(), np, s));
        count_launch(2);
        int64_t nu = 0;
        GBK_CUDA(cudaMemcpyAsync(&nu, nsel, 8, cudaMemcpyDeviceToHost, s));
        GBK_CUDA(cudaStreamSynchronize(s));
        // drop the zero sums (keys and values compacted by the same flags)
        {
            unsigned long long* kk = nullptr;
            T* vv = nullptr;
            if (!need(dev.get(&kk, 8 * std::max<int64_t>(nu, 1))) || !need(dev.get(&vv, sizeof(T) * std::max<int64_t>(nu, 1)))) {
                set_error("gbk_mxm: out of device memory for a block's result");
                return GBK_OUT_OF_MEMORY;
            }
            okeys.push_back(kk);
            ovals.push_back(vv);
            orow0.push_back(cuts[c]);
            tb = tbytes;
            GBK_CUDA(cub::DeviceSelect::If(tmp, tb, val, vv, nsel, nu, NonZero<T>(), s));
            count_launch(1);
            // the same selection for the keys: flags from the values
            k_nonzero_flags<T><<<nb(nu), 256, 0, s>>>(val, nu, flag);
            GBK_LAUNCHED();
            tb = tbytes;
            GBK_CUDA(cub::DeviceSelect::Flagged(tmp, tb, key, flag, kk, nsel + 1, nu, s));
            count_launch(1);
            int64_t kept[2] = {0, 0};
            GBK_CUDA(cudaMemcpyAsync(kept, nsel, 16, cudaMemcpyDeviceToHost, s));
            GBK_CUDA(cudaStreamSynchronize(s));
            ocnt.push_back(kept[0]);
            total += kept[0];
        }
    }
    GBK_REQUIRE(total < INT32_MAX, GBK_INVALID_VALUE, "gbk_mxm: the product has %lld entries (int32 limit)",
                (long long)total);
    // CSR of the result
    int32_t *row = nullptr, *col = nullptr, *ptr = nullptr;
    T* cval = nullptr;
    if (!need(dev.get(&row, 4 * total)) || !need(dev.get(&col, 4 * total)) || !need(dev.get(&ptr, 4 * (n + 1))) ||
        !need(dev.get(&cval, sizeof(T) * total))) {
        set_error("gbk_mxm: out of device memory for the result");
        return GBK_OUT_OF_MEMORY;
    }
    int64_t at = 0;
    for (size_t c = 0; c < okeys.size(); ++c) {
        if (ocnt[c] > 0) {
            k_split_keys<<<nb(ocnt[c]), 256, 0, s>>>(okeys[c], ocnt[c], (int32_t)orow0[c], colbits, row + at, col + at);
            GBK_LAUNCHED();
            GBK_CUDA(cudaMemcpyAsync(cval + at, ovals[c], sizeof(T) * ocnt[c], cudaMemcpyDeviceToDevice, s));
        }
        at += ocnt[c];
    }
    k_bounds<<<nb(total + 1), 256, 0, s>>>(row, total, n, ptr);
    GBK_LAUNCHED();
    GBK_CUDA(cudaStreamSynchronize(s));
    return gbk_matrix_create_csr(out, n, m, total, ptr, col, cval, std::is_same<T, float>::value ? GBK_F32 : GBK_I32,
                                 1, s);
}

// ---------------------------------------------------------------------------
// triangle counting

// The count needs each undirected edge once, from its (degree, id)-smaller end
// (u, v): the triangles are the common entries of N+(u) and N+(v).  On an
// R-MAT graph of 2^17 vertices no N+ list is longer than 315 entries although
// the largest degree is 15,743, so every list fits a small hash table in
// shared memory.  The preparation works on tiles of 256 consecutive entries
// (a warp each), never on rows: with a thread per row the one thread on a hub
// row took 1.1 - 1.3 ms in each of two kernels where all of the preparation
// now takes 45 us (same graph).
constexpr int kTcTile = 256;

enum { kTcAsymmetric = 1, kTcLoop = 2, kTcDuplicate = 4 };

// deg: row lengths; tile_row: the row of each tile's first entry (n - 1 past
// the last); *bad gets kTcAsymmetric where A's and the CSC's row starts differ.
__global__ void __launch_bounds__(256) k_tc_degrees(const int32_t* __restrict__ ap, const int32_t* __restrict__ tp,
                                                    int64_t n, int64_t ntiles, int32_t* __restrict__ deg,
                                                    int32_t* __restrict__ tile_row, int* __restrict__ bad) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool diff = i <= n && ap[i] != tp[i];
    if (i < n) {
        const int32_t b = ap[i], d = ap[i + 1] - b;
        deg[i] = d;
        const int64_t end = (int64_t)b + d;
        for (int64_t t = ((int64_t)b + kTcTile - 1) / kTcTile; t * kTcTile < end; ++t) tile_row[t] = (int32_t)i;
        if (i == n - 1) tile_row[ntiles] = (int32_t)i;
    }
    if (__any_sync(0xffffffffu, diff) && (threadIdx.x & 31) == 0) atomicOr(bad, kTcAsymmetric);
}

// Marks the oriented entries, one bit each (marks) and their number per tile
// (cnt; cnt[ntiles] = 0), and checks the pattern: *bad collects kTcAsymmetric
// (A differs from its CSC), kTcLoop (a diagonal entry) and kTcDuplicate (an
// entry equal to the one before it in its row).  Each lane searches the rows
// of its eight entries between the rows of the tile's ends, four independent
// searches at a time over a few neighbouring row starts.
__global__ void __launch_bounds__(256) k_tc_mark(const int32_t* __restrict__ ap, const int32_t* __restrict__ ai,
                                                 const int32_t* __restrict__ ti, const int32_t* __restrict__ deg,
                                                 const int32_t* __restrict__ tile_row, int64_t nnz, int64_t ntiles,
                                                 uint32_t* __restrict__ marks, int32_t* __restrict__ cnt,
                                                 int* __restrict__ bad) {
    constexpr int kSubs = kTcTile / 32, kHalf = kSubs / 2;
    const int lane = threadIdx.x & 31;
    const int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= ntiles) return;  // the whole warp leaves together
    // the last row with ap[row] <= e lies in [first, last]
    const int32_t first = tile_row[t], last = tile_row[t + 1];
    int f = 0;
    int32_t kept = 0, word = 0;
    for (int h = 0; h < 2; ++h) {
        const int64_t e0 = t * kTcTile + 32 * kHalf * h + lane;
        int32_t c[kHalf], dv[kHalf], lo[kHalf], hi[kHalf];
#pragma unroll
        for (int i = 0; i < kHalf; ++i) {
            const int64_t e = e0 + 32 * i;
            c[i] = e < nnz ? ai[e] : -1;
            if (e < nnz && ti[e] != c[i]) f |= kTcAsymmetric;
        }
#pragma unroll
        for (int i = 0; i < kHalf; ++i) {
            dv[i] = c[i] >= 0 ? __ldg(deg + c[i]) : 0;
            lo[i] = first;
            hi[i] = last;
        }
        for (int32_t span = last - first; span > 0; span >>= 1) {  // the range halves (rounded down) each step
#pragma unroll
            for (int i = 0; i < kHalf; ++i)
                if (lo[i] < hi[i]) {
                    const int32_t mid = lo[i] + ((hi[i] - lo[i] + 1) >> 1);
                    if (__ldg(ap + mid) <= e0 + 32 * i)
                        lo[i] = mid;
                    else
                        hi[i] = mid - 1;
                }
        }
#pragma unroll
        for (int i = 0; i < kHalf; ++i) {
            const int64_t e = e0 + 32 * i;
            bool keep = false;
            int32_t before = __shfl_up_sync(0xffffffffu, c[i], 1);
            if (lane == 0 && e > 0 && e < nnz) before = ai[e - 1];
            if (c[i] >= 0) {
                const int32_t u = lo[i], du = __ldg(deg + u);
                if (c[i] == u) f |= kTcLoop;
                if (before == c[i] && e > __ldg(ap + u)) f |= kTcDuplicate;
                keep = du < dv[i] || (du == dv[i] && u < c[i]);
            }
            const unsigned m = __ballot_sync(0xffffffffu, keep);
            kept += __popc(m);
            if (lane == kHalf * h + i) word = (int32_t)m;
        }
    }
    if (lane < kSubs) marks[t * kSubs + lane] = (uint32_t)word;
    if (lane == 0) {
        cnt[t] = kept;
        if (t == 0) cnt[ntiles] = 0;
    }
    f = __reduce_or_sync(0xffffffffu, f);
    if (lane == 0 && f) atomicOr(bad, f);
}

// Oriented entries before entry e (e <= nnz).
__device__ __forceinline__ int32_t tc_rank(const uint32_t* __restrict__ marks, const int32_t* __restrict__ base,
                                           int64_t nnz, int32_t e) {
    const int32_t t = e / kTcTile;
    int32_t r = base[t];
    if (e < nnz) {
        const uint32_t* w = marks + (int64_t)t * (kTcTile / 32);
        const int in = e % kTcTile;
        for (int i = 0; i < in / 32; ++i) r += __popc(w[i]);
        r += __popc(w[in / 32] & ((1u << (in % 32)) - 1u));
    } else if (e % kTcTile) {
        r = base[t + 1];
    }
    return r;
}

// The work items of the count.  An edge {v, w} belongs to its end with the
// longer oriented list (ties: the larger id), v: N+(v) becomes a set in shared
// memory and the entries of N+(w) are looked up in it, so the lookups are the
// sum of min(|N+(v)|, |N+(w)|) over the edges (128 M on R-MAT 2^17; with the
// edge always at its source 252 M).  An item is a vertex v and a run of at
// most `run` entries of its row, whose ends w it takes the eligible ones of:
// hub rows are spread over many items.  Classes by |N+(v)|: up to 32 a warp
// per item; above that a CTA per item, on a bitmap over all vertices while
// that fits shared memory, otherwise on hash tables of 4096 and 32768 slots,
// and by search in the list itself above 8192 entries.
constexpr int kTcClasses = 4;
constexpr int kTcWarpRun = 128, kTcCtaRun = 256;

struct TcItems {
    int2* v[kTcClasses];         // (vertex, first entry)
    int32_t most[kTcClasses];    // largest |N+(v)| of the class
    int32_t run[kTcClasses];     // entries per item
};

// op (row starts of the oriented lists) and the items of each class.
__global__ void __launch_bounds__(256) k_tc_rows(const int32_t* __restrict__ ap, int64_t n, int64_t nnz,
                                                 const uint32_t* __restrict__ marks, const int32_t* __restrict__ base,
                                                 const int* __restrict__ bad, int32_t* __restrict__ op, TcItems items,
                                                 int32_t* __restrict__ nitem) {
    if (*bad & (kTcAsymmetric | kTcLoop)) return;
    const int lane = threadIdx.x & 31;
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int cls = -1;
    int32_t ab = 0, ae = 0;
    if (v < n) {
        ab = ap[v];
        ae = ap[v + 1];
        const int32_t b = tc_rank(marks, base, nnz, ab), e = tc_rank(marks, base, nnz, ae);
        op[v] = b;
        if (v == n - 1) op[n] = e;
        if (e - b >= 2)
            for (cls = 0; e - b > items.most[cls]; ++cls) {}
    }
    for (int c = 0; c < kTcClasses; ++c) {
        const int32_t run = items.run[c];
        const int32_t cnt = cls == c ? (int32_t)(((int64_t)ae - ab + run - 1) / run) : 0;
        int32_t incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const int32_t all = __shfl_sync(0xffffffffu, incl, 31);
        if (!all) continue;
        int32_t at = 0;
        if (lane == 0) at = atomicAdd(nitem + c, all);
        at = __shfl_sync(0xffffffffu, at, 0) + incl - cnt;
        for (int32_t i = 0; i < cnt; ++i) items.v[c][at + i] = make_int2((int32_t)v, ab + i * run);
    }
}

// oi: the oriented entries' columns, in entry order (a warp per tile).
__global__ void __launch_bounds__(256) k_tc_fill(const int32_t* __restrict__ ai, int64_t nnz, int64_t ntiles,
                                                 const uint32_t* __restrict__ marks, const int32_t* __restrict__ base,
                                                 const int* __restrict__ bad, int32_t* __restrict__ oi) {
    if (*bad & (kTcAsymmetric | kTcLoop)) return;  // oi has room for the half that a simple graph keeps
    const int lane = threadIdx.x & 31;
    const int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= ntiles) return;
    int32_t at = base[t];
#pragma unroll
    for (int sub = 0; sub < kTcTile / 32; ++sub) {
        const uint32_t m = marks[t * (kTcTile / 32) + sub];
        if ((m >> lane) & 1u) oi[at + __popc(m & ((1u << lane) - 1u))] = ai[t * kTcTile + 32 * sub + lane];
        at += __popc(m);
    }
}

// The sets N+(v) is looked up in.  Each is built and cleared by `nt` threads,
// thread t, over the list l[0, d).

// Open addressing over int32 slots (-1 empty), at least four per entry: a
// lookup that misses ends after 1.4 slots on average.
struct TcHash {
    int32_t* tab;
    uint32_t mask;
    int shift;
    __device__ void build(const int32_t* __restrict__ l, int32_t d, int t, int nt) {
        const int lg = max(6, 32 - __clz(4 * d - 1));
        mask = (1u << lg) - 1u;
        shift = 32 - lg;
        for (int k = t; k <= (int)mask; k += nt) tab[k] = -1;
        if (nt == 32) __syncwarp();
        else __syncthreads();
        for (int32_t j = t; j < d; j += nt)
            for (uint32_t h = slot(l[j]);; h = (h + 1) & mask) {
                const int32_t old = atomicCAS(tab + h, -1, l[j]);
                if (old == -1 || old == l[j]) break;
            }
    }
    __device__ void clear(const int32_t*, int32_t, int, int) {}
    __device__ __forceinline__ uint32_t slot(int32_t key) const { return ((uint32_t)key * 0x9E3779B1u) >> shift; }
    __device__ __forceinline__ bool has(int32_t key) const {
        for (uint32_t h = slot(key);; h = (h + 1) & mask) {
            const int32_t x = tab[h];
            if (x == key) return true;
            if (x < 0) return false;
        }
    }
};

// One bit per vertex (all clear between items).  A lookup is one load whatever
// the keys, where the hash table's slowest lane sets the pace.  The words of a
// 32-word group are permuted by the higher bits, so that the hub ids of R-MAT
// graphs (few bits set) spread over the banks.
struct TcBits {
    uint32_t* w;
    __device__ void build(const int32_t* __restrict__ l, int32_t d, int t, int nt) {
        for (int32_t j = t; j < d; j += nt) atomicOr(w + word(l[j]), 1u << (l[j] & 31));
    }
    __device__ void clear(const int32_t* __restrict__ l, int32_t d, int t, int nt) {
        for (int32_t j = t; j < d; j += nt) w[word(l[j])] = 0;
    }
    __device__ __forceinline__ int32_t word(int32_t key) const { return (key >> 5) ^ ((key >> 10) & 31); }
    __device__ __forceinline__ bool has(int32_t key) const { return (w[word(key)] >> (key & 31)) & 1u; }
};

// The sorted list itself.
struct TcSearch {
    const int32_t* l;
    int32_t d;
    __device__ void build(const int32_t* __restrict__ list, int32_t len, int, int) {
        l = list;
        d = len;
    }
    __device__ void clear(const int32_t*, int32_t, int, int) {}
    __device__ __forceinline__ bool has(int32_t key) const {
        int32_t lo = 0, hi = d;
        while (lo < hi) {
            const int32_t mid = (lo + hi) >> 1;
            if (l[mid] < key)
                lo = mid + 1;
            else
                hi = mid;
        }
        return lo < d && l[lo] == key;
    }
};

// The eligible ends among 32 row entries (w per lane, -1 none): the entries of
// their oriented lists found in the set of v (d entries).  Each quarter of the
// warp walks its own lists, 32 entries (four per lane) at a step, and goes on
// to its next list by itself, so short lists cost an eighth of a warp each and
// four loads are in flight per lane (R-MAT 2^17: 237 us for k_tc_cta; with the
// whole warp on one list and one load at a time 355 us).  `slots`: 32 list
// ranges of the warp.
template <class Set>
__device__ __forceinline__ uint32_t tc_lookup(const Set& set, const int32_t* __restrict__ op,
                                              const int32_t* __restrict__ oi, int32_t v, int32_t d, int32_t w, int lane,
                                              int2* slots) {
    constexpr unsigned kAllLanes = 0xffffffffu;
    const int32_t wb = w >= 0 ? __ldg(op + w) : 0, we = w >= 0 ? __ldg(op + w + 1) : 0;
    const int32_t dw = we - wb;
    const bool mine = dw > 0 && (dw < d || (dw == d && w < v));
    const unsigned todo = __ballot_sync(kAllLanes, mine);
    const int nl = __popc(todo);
    if (mine) slots[__popc(todo & ((1u << lane) - 1u))] = make_int2(wb, we);
    __syncwarp();
    uint32_t c = 0;
    int32_t p = 0, e = 0;  // what is left of the quarter's current list
    for (int at = lane >> 3;;) {
        if (p >= e && at < nl) {
            p = slots[at].x;
            e = slots[at].y;
            at += 4;
        }
        if (!__any_sync(kAllLanes, p < e)) break;
        int32_t key[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int32_t q = p + 8 * i + (lane & 7);
            key[i] = q < e ? __ldg(oi + q) : -1;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (key[i] >= 0) c += set.has(key[i]);
        p += 32;
    }
    __syncwarp();
    return c;
}

// The CTA's counts into *total with one atomic.
template <int THREADS>
__device__ __forceinline__ void tc_add_total(unsigned long long mine, unsigned long long* total) {
    __shared__ unsigned long long part[THREADS / 32];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mine += __shfl_down_sync(0xffffffffu, mine, off);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < THREADS / 32; ++w) mine += part[w];
        if (mine) atomicAdd(total, mine);
    }
}

struct TcArgs {
    const int32_t* ap;
    const int32_t* ai;
    const int32_t* op;
    const int32_t* oi;
    const int2* items;
    const int32_t* nitem;
    const int* bad;
    unsigned long long* total;
    int32_t* next;  // the next item to hand out
    int32_t run;
    int32_t words;  // of the bitmap
};

// A warp per item (|N+(v)| <= 32).
__global__ void __launch_bounds__(256, 8) k_tc_warp(TcArgs a) {
    __shared__ int32_t tabs[8][128];
    __shared__ int2 s_slots[8][32];
    if (*a.bad) return;
    int2* slots = s_slots[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    TcHash set;
    set.tab = tabs[threadIdx.x >> 5];
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int32_t ni = *a.nitem;
    unsigned long long mine = 0;
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < ni; i += nw) {
        const int2 it = a.items[i];
        const int32_t b = a.op[it.x], d = a.op[it.x + 1] - b;
        const int32_t* __restrict__ row = a.ai + it.y;
        const int32_t len = min(a.ap[it.x + 1] - it.y, a.run);
        set.build(a.oi + b, d, lane, 32);
        __syncwarp();
        for (int32_t e = 0; e < len; e += 32)
            mine += tc_lookup(set, a.op, a.oi, it.x, d, e + lane < len ? row[e + lane] : -1, lane, slots);
        __syncwarp();
    }
    tc_add_total<256>(mine, a.total);
}

// A CTA per item, items and the 32-entry groups inside them handed out by
// counters (with vertices in order the CTAs were idle for 28 % of the time, and
// with equal shares of an item its warps waited at the barrier).  Bound by the
// lookups (a list entry from L2, then a random shared-memory word): R-MAT 2^17
// 237 us, and 30 us for k_tc_warp, where a warp per edge with a binary search
// per entry of the shorter list took 920 us.
template <class Set, int THREADS>
__global__ void __launch_bounds__(THREADS, 2048 / THREADS) k_tc_cta(TcArgs a) {
    extern __shared__ uint32_t smem[];
    __shared__ int32_t s_item[2], s_group;
    __shared__ int2 s_slots[THREADS / 32][32];
    if (*a.bad) return;
    int2* slots = s_slots[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    Set set;
    if constexpr (std::is_same<Set, TcHash>::value) set.tab = (int32_t*)smem;
    if constexpr (std::is_same<Set, TcBits>::value) {
        set.w = smem;
        for (int i = threadIdx.x; i < a.words; i += THREADS) smem[i] = 0;
    }
    const int32_t ni = *a.nitem;
    unsigned long long mine = 0;
    if (threadIdx.x == 0) s_item[0] = atomicAdd(a.next, 1);
    for (int turn = 0;; turn ^= 1) {
        __syncthreads();  // the item is known, the set clear
        const int32_t i = s_item[turn];
        if (i >= ni) break;
        const int2 it = a.items[i];
        const int32_t b = a.op[it.x], d = a.op[it.x + 1] - b;
        const int32_t* __restrict__ row = a.ai + it.y;
        const int32_t len = min(a.ap[it.x + 1] - it.y, a.run);
        if (threadIdx.x == 0) {
            s_item[turn ^ 1] = atomicAdd(a.next, 1);
            s_group = 0;
        }
        set.build(a.oi + b, d, threadIdx.x, THREADS);
        __syncthreads();
        for (;;) {
            int32_t g = 0;
            if (lane == 0) g = atomicAdd(&s_group, 1);
            const int32_t e = 32 * __shfl_sync(0xffffffffu, g, 0);
            if (e >= len) break;
            mine += tc_lookup(set, a.op, a.oi, it.x, d, e + lane < len ? row[e + lane] : -1, lane, slots);
        }
        __syncthreads();
        set.clear(a.oi + b, d, threadIdx.x, THREADS);
    }
    tc_add_total<THREADS>(mine, a.total);
}

// Patterns with repeated entries: a repeated entry of an edge's shorter list
// counts each time it is listed (and the longer list's only once), so which
// list is walked decides the count, and it is the shorter one for every edge.
__global__ void __launch_bounds__(256) k_tc_duplicates(const int32_t* __restrict__ op, const int32_t* __restrict__ oi,
                                                       const int32_t* __restrict__ orow, int64_t m,
                                                       unsigned long long* __restrict__ total) {
    const int lane = threadIdx.x & 31;
    const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    unsigned long long mine = 0;
    for (int64_t e = gw; e < m; e += nw) {
        int32_t u = orow[e], v = oi[e];
        if (op[u + 1] - op[u] > op[v + 1] - op[v]) {
            const int32_t x = u;
            u = v;
            v = x;
        }
        TcSearch longer;
        longer.build(oi + op[v], op[v + 1] - op[v], 0, 0);
        for (int32_t p = op[u] + lane; p < op[u + 1]; p += 32) mine += longer.has(oi[p]);
    }
    tc_add_total<256>(mine, total);
}

}  // namespace

}  // namespace gbk

using namespace gbk;

extern "C" int gbk_triangle_count(gbk_matrix A, uint64_t* count, void* stream) {
    GBK_REQUIRE(A && count, GBK_NULL_POINTER, "gbk_triangle_count: NULL argument");
    GBK_REQUIRE(A->csr.nrows == A->csr.ncols, GBK_DIMENSION_MISMATCH, "gbk_triangle_count: A is not square");
    cudaStream_t s = (cudaStream_t)stream;
    int rc = ensure_csc(A, s);
    if (rc) return rc;
    const CsrView& a = A->csr;
    const CsrView& t = A->csc;
    const int64_t n = a.nrows, nnz = a.nnz;
    if (nnz == 0) {
        *count = 0;
        return GBK_SUCCESS;
    }
    // Everything up to the count is queued before the one read-back: the
    // kernels after k_tc_mark look at its verdict on the device.
    const int64_t ntiles = (nnz + kTcTile - 1) / kTcTile;
    StreamScratch dev(s);
    uint8_t* mem = nullptr;  // bad, class counts, total, then the arrays
    size_t tb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb, (int32_t*)nullptr, (int32_t*)nullptr, ntiles + 1, s);
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t b_marks = up(4 * (size_t)ntiles * (kTcTile / 32)), b_cnt = up(4 * (size_t)(ntiles + 1)),
                 b_op = up(4 * (size_t)(n + 1)), b_oi = up(4 * (size_t)(nnz / 2 + 1));
    // The bitmap serves up to 2^18 vertices (32 KB, six CTAs on an SM); with
    // more, too few CTAs fit and the hash tables are as fast or faster (whole
    // call, R-MAT 2^18: 0.91 ms against 1.22 with hash tables, 2^19: 2.35
    // against 2.21, 2^20: 12.3 against 5.1).
    const int64_t words = (n + 1023) / 1024 * 32;
    const bool bits = words <= 8192;
    TcItems items;
    const int32_t most[kTcClasses] = {32, bits ? INT_MAX : 1024, bits ? INT_MAX : 8192, INT_MAX};
    size_t b_items[kTcClasses], b_all = 0;
    for (int c = 0; c < kTcClasses; ++c) {
        items.most[c] = most[c];
        items.run[c] = c == 0 ? kTcWarpRun : kTcCtaRun;
        // one item per started run: vertices whose lists are longer than the
        // class below's share nnz / 2 oriented entries
        const int64_t least = c == 0 ? 2 : (int64_t)most[c - 1] + 1;
        b_items[c] = up(8 * (size_t)(std::min<int64_t>(n, nnz / 2 / least + 1) + nnz / items.run[c] + 1));
        if (c > 0 && most[c - 1] == INT_MAX) b_items[c] = 256;
        b_all += b_items[c];
    }
    if (dev.get(&mem, 256 + b_marks + 2 * b_cnt + b_op + b_all + b_oi + up(tb))) {
        set_error("gbk_triangle_count: out of device memory");
        return GBK_OUT_OF_MEMORY;
    }
    int* bad = (int*)mem;
    int32_t* nitem = (int32_t*)(mem + 16);
    unsigned long long* total = (unsigned long long*)(mem + 64);
    int32_t* next = (int32_t*)(mem + 128);
    uint8_t* at = mem + 256;
    auto take = [&](size_t bytes) {
        uint8_t* p = at;
        at += bytes;
        return p;
    };
    uint32_t* marks = (uint32_t*)take(b_marks);
    int32_t* cnt = (int32_t*)take(b_cnt);
    int32_t* base = (int32_t*)take(b_cnt);
    int32_t* op = (int32_t*)take(b_op);
    for (int c = 0; c < kTcClasses; ++c) items.v[c] = (int2*)take(b_items[c]);
    int32_t* oi = (int32_t*)take(b_oi);
    void* tmp = take(up(tb));
    GBK_CUDA(cudaMemsetAsync(mem, 0, 256, s));
    const unsigned gt = (unsigned)((ntiles + 7) / 8);
    int32_t* deg = op;  // until k_tc_rows writes the row starts
    int32_t* tile_row = base;  // until the scan
    k_tc_degrees<<<nb(n + 1), 256, 0, s>>>(a.ptr, t.ptr, n, ntiles, deg, tile_row, bad);
    GBK_LAUNCHED();
    k_tc_mark<<<gt, 256, 0, s>>>(a.ptr, a.idx, t.idx, deg, tile_row, nnz, ntiles, marks, cnt, bad);
    GBK_LAUNCHED();
    GBK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, cnt, base, ntiles + 1, s));
    count_launch(1);
    k_tc_rows<<<nb(n), 256, 0, s>>>(a.ptr, n, nnz, marks, base, bad, op, items, nitem);
    GBK_LAUNCHED();
    k_tc_fill<<<gt, 256, 0, s>>>(a.idx, nnz, ntiles, marks, base, bad, oi);
    GBK_LAUNCHED();
    auto args = [&](int c) {
        return TcArgs{a.ptr, a.idx, op, oi, items.v[c], nitem + c, bad, total, next + c, items.run[c], (int32_t)words};
    };
    auto launch_cta = [&](auto kern, int threads, int per_sm, int smem, int c) -> int {
        GBK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        kern<<<(unsigned)(num_sms() * per_sm), threads, smem, s>>>(args(c));
        GBK_LAUNCHED();
        return GBK_SUCCESS;
    };
    // a list of d entries ends at d vertices of at least as many entries, so
    // nnz >= d (d + 1): small graphs cannot reach the larger classes
    auto reached = [&](int c) { return nnz > ((int64_t)most[c - 1] + 1) * ((int64_t)most[c - 1] + 1); };
    int rc2 = GBK_SUCCESS;
    if (bits) {
        if (reached(1))
            rc2 = launch_cta(k_tc_cta<TcBits, 256>, 256, 8, (int)words * 4, 1);
    } else {
        if (reached(3)) rc2 = launch_cta(k_tc_cta<TcSearch, 256>, 256, 8, 0, 3);
        if (!rc2 && reached(2)) rc2 = launch_cta(k_tc_cta<TcHash, 1024>, 1024, 1, 4 * 32768, 2);
        if (!rc2 && reached(1)) rc2 = launch_cta(k_tc_cta<TcHash, 256>, 256, 8, 4 * 4096, 1);
    }
    if (rc2) return rc2;
    k_tc_warp<<<(unsigned)std::min<int64_t>((n + 7) / 8, (int64_t)num_sms() * 8), 256, 0, s>>>(args(0));
    GBK_LAUNCHED();
    struct {
        int bad;
        int pad[15];
        unsigned long long total;
    } head{};
    const int rb = read_back(&head, mem, sizeof(head), s);
    if (rb) return rb;
    if (head.bad & (kTcAsymmetric | kTcLoop)) {
        // not a simple undirected graph: Burkhardt's sum (sum ((A * A) .* A)) / 6 as it stands
        gbk_matrix C = nullptr;
        rc = gbk_mxm_masked(&C, A, A, A, GBK_PLUS_ONE, GBK_I32, stream);
        if (rc) return rc;
        const CsrView& c = C->csr;
        void* rtmp = nullptr;
        size_t rtb = 0;
        long long* sum = nullptr;
        rc = dev.get(&sum, 8);
        if (!rc) {
            cub::DeviceReduce::Sum(nullptr, rtb, (const int32_t*)c.val, sum, c.nnz, s);
            rc = dev.get(&rtmp, rtb);
        }
        long long hs = 0;
        if (!rc && cub::DeviceReduce::Sum(rtmp, rtb, (const int32_t*)c.val, sum, c.nnz, s) == cudaSuccess &&
            cudaMemcpyAsync(&hs, sum, 8, cudaMemcpyDeviceToHost, s) == cudaSuccess &&
            cudaStreamSynchronize(s) == cudaSuccess) {
            count_launch(1);
            *count = (uint64_t)(hs / 6);
        } else if (!rc) {
            rc = cuda_fail(cudaGetLastError(), "triangle count reduce", __FILE__, __LINE__);
        }
        gbk_matrix_destroy(C);
        return rc;
    }
    if (head.bad & kTcDuplicate) {
        int32_t m = 0;
        int32_t* orow = nullptr;
        GBK_CUDA(cudaMemcpyAsync(&m, op + n, 4, cudaMemcpyDeviceToHost, s));
        GBK_CUDA(cudaStreamSynchronize(s));
        if (dev.get(&orow, 4 * (int64_t)m)) return GBK_OUT_OF_MEMORY;
        if (m > 0) {
            k_entry_rows<<<nb(m), 256, 0, s>>>(op, n, m, orow);
            GBK_LAUNCHED();
            k_tc_duplicates<<<(unsigned)std::min<int64_t>((m + 7) / 8, (int64_t)num_sms() * 8), 256, 0, s>>>(op, oi, orow,
                                                                                                      m, total);
            GBK_LAUNCHED();
        }
        GBK_CUDA(cudaMemcpyAsync(&head.total, total, 8, cudaMemcpyDeviceToHost, s));
        GBK_CUDA(cudaStreamSynchronize(s));
    }
    *count = head.total;
    return GBK_SUCCESS;
}

extern "C" int gbk_mxm(gbk_matrix* out, gbk_matrix A, gbk_matrix B, gbk_semiring sr, void* stream) {
    GBK_REQUIRE(out && A && B, GBK_NULL_POINTER, "gbk_mxm: NULL argument");
    GBK_REQUIRE(A->vtype == B->vtype, GBK_DOMAIN_MISMATCH, "gbk_mxm: A and B value types differ");
    GBK_REQUIRE(A->csr.ncols == B->csr.nrows, GBK_DIMENSION_MISMATCH, "gbk_mxm: A is %lldx%lld, B %lldx%lld",
                (long long)A->csr.nrows, (long long)A->csr.ncols, (long long)B->csr.nrows, (long long)B->csr.ncols);
    cudaStream_t s = (cudaStream_t)stream;
    bool done = false;
    // a windowed entry takes 8 bytes of scratch, an expanded product 24
    const int rc = mxm_window(out, A->csr, B->csr, A->vtype, sr, 3 * block_products(), &done, s);
    if (rc || done) return rc;
#define MXM_CASE(SRV)                                                                                 \
    case SRV:                                                                                         \
        return A->vtype == GBK_F32 ? mxm_unmasked<SRV, float>(out, A->csr, B->csr, s)                 \
                                   : mxm_unmasked<SRV, int32_t>(out, A->csr, B->csr, s);
    switch (sr) {
        MXM_CASE(GBK_PLUS_TIMES)
        MXM_CASE(GBK_PLUS_SECOND)
        MXM_CASE(GBK_PLUS_ONE)
        MXM_CASE(GBK_MIN_PLUS)
        MXM_CASE(GBK_MIN_SECOND)
        MXM_CASE(GBK_LOR_LAND)
        default:
            set_error("gbk_mxm: semiring %d not provided (plus-times, plus-second, plus-one, min-plus, "
                      "min-second, or-and)",
                      (int)sr);
            return GBK_UNSUPPORTED;
    }
#undef MXM_CASE
}

extern "C" int gbk_mxm_masked(gbk_matrix* out, gbk_matrix M, gbk_matrix A, gbk_matrix B, gbk_semiring sr,
                              gbk_dtype ctype, void* stream) {
    GBK_REQUIRE(out && M && A && B, GBK_NULL_POINTER, "gbk_mxm_masked: NULL argument");
    GBK_REQUIRE(sr == GBK_PLUS_ONE || sr == GBK_PLUS_TIMES, GBK_UNSUPPORTED,
                "gbk_mxm_masked: semiring %d not provided (GBK_PLUS_ONE, GBK_PLUS_TIMES)", (int)sr);
    GBK_REQUIRE(ctype == GBK_I32 || ctype == GBK_F32, GBK_UNSUPPORTED, "gbk_mxm_masked: output type %d", (int)ctype);
    GBK_REQUIRE(A->vtype == B->vtype, GBK_DOMAIN_MISMATCH, "gbk_mxm_masked: A and B value types differ");
    GBK_REQUIRE(A->csr.ncols == B->csr.nrows && M->csr.nrows == A->csr.nrows && M->csr.ncols == B->csr.ncols,
                GBK_DIMENSION_MISMATCH, "gbk_mxm_masked: dimensions do not agree");
    cudaStream_t s = (cudaStream_t)stream;
    int rc = ensure_csc(B, s);
    if (rc) return rc;
    const CsrView& m = M->csr;
    const CsrView& a = A->csr;
    const CsrView& b = B->csc;
    void* vals = nullptr;  // from the stream-ordered pool: results of this size recur (triangle counting)
    GBK_CUDA(cudaMallocAsync(&vals, 4 * (m.nnz > 0 ? m.nnz : 1), s));
    if (m.nnz > 0) {
        const int threads = 256;
        int64_t groups = (m.nnz + 31) / 32;
        int64_t blocks = (groups * 32 + threads - 1) / threads;
        int64_t cap = (int64_t)num_sms() * 16;
        if (blocks > cap) blocks = cap;
#define SPGEMM_LAUNCH(SRV, CT, AT)                                                                              \
    k_masked_spgemm<SRV, CT, AT><<<(unsigned)blocks, threads, 0, s>>>(m.ptr, m.idx, m.nrows, m.nnz, a.ptr, a.idx, \
                                                                      (const AT*)a.val, b.ptr, b.idx,           \
                                                                      (const AT*)b.val, (CT*)vals)
        if (A->vtype == GBK_F32) {
            if (sr == GBK_PLUS_ONE) {
                if (ctype == GBK_I32) SPGEMM_LAUNCH(GBK_PLUS_ONE, int32_t, float);
                else SPGEMM_LAUNCH(GBK_PLUS_ONE, float, float);
            } else {
                if (ctype == GBK_I32) SPGEMM_LAUNCH(GBK_PLUS_TIMES, int32_t, float);
                else SPGEMM_LAUNCH(GBK_PLUS_TIMES, float, float);
            }
        } else {
            if (sr == GBK_PLUS_ONE) {
                if (ctype == GBK_I32) SPGEMM_LAUNCH(GBK_PLUS_ONE, int32_t, int32_t);
                else SPGEMM_LAUNCH(GBK_PLUS_ONE, float, int32_t);
            } else {
                if (ctype == GBK_I32) SPGEMM_LAUNCH(GBK_PLUS_TIMES, int32_t, int32_t);
                else SPGEMM_LAUNCH(GBK_PLUS_TIMES, float, int32_t);
            }
        }
#undef SPGEMM_LAUNCH
        GBK_LAUNCHED();
    }
    GBK_CUDA(cudaStreamSynchronize(s));
    rc = gbk_matrix_create_csr(out, m.nrows, m.ncols, m.nnz, m.ptr, m.idx, vals, ctype, 1, stream);
    cudaFreeAsync(vals, s);
    return rc;
}
