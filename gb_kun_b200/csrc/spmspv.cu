// Push SpMSpV and sparse-mask SpMV.
//
// SpMSpV replaces backend::SpMSpV with its three push kernels
// (src/backend/spmspv/spmspv.h:103-158, spmspv_atomics.h:5-170): for every
// frontier entry (i, x_i) scatter mul(A, x_i) into y.  The reference gives
// each OpenMP thread frontier vertices and updates y with `omp atomic`,
// plain stores or an `omp critical` section per edge.  Here a warp takes 8 or
// 32 frontier entries and spreads the edges of their rows under kHeavyRow
// entries over its lanes; longer rows are cut into kPiece-entry pieces that a
// second kernel hands out one per warp, so a hub is spread over many warps.
// (The first form scanned the frontier's degrees, copied y and masked it in a
// pass of its own: nine operations on the stream and four allocations, which
// took longer than the pushes.  Or-and from 3 % of the vertices of an R-MAT
// graph of 2^20, masked: 56 -> 25 us.)  Updates are
// warp-aggregated: lanes whose edges hit the same output element (match-any on
// the index) combine their values with the semiring's add in a tree over the
// group, and one lane per group issues the atomic (add; min on integers, a CAS
// loop on floats).  Or-monoids store 1 without an atomic, as the reference
// does, and read neither values nor frontier values.
#include <algorithm>

#include "common.cuh"
#include "internal.h"

namespace gbk {

namespace {

constexpr int kPushThreads = 256;

__device__ __forceinline__ void atomic_min_val(int32_t* p, int32_t v) { atomicMin(p, v); }
__device__ __forceinline__ void atomic_min_val(float* p, float v) {
    int32_t* ip = (int32_t*)p;
    int32_t old = *ip;
    while (v < __int_as_float(old)) {
        int32_t prev = atomicCAS(ip, old, __float_as_int(v));
        if (prev == old) break;
        old = prev;
    }
}

// Bit position of the r-th (0-based) set bit of m (m has more than r bits).
__device__ __forceinline__ int nth_set_bit(unsigned m, int r) {
    int pos = 0;
#pragma unroll
    for (int w = 16; w >= 1; w >>= 1)
        if (__popc(m & ((1u << (pos + w)) - 1u)) <= r) pos += w;
    return pos;
}

// What a push does to y[j], by the semiring's add(3, 5) (semiring_probe).
enum { kPushAdd, kPushOne, kPushMin, kPushNothing };
template <int SR>
constexpr int push_kind() {
    if (SR == GBK_PLUS_TIMES || SR == GBK_PLUS_SECOND || SR == GBK_PLUS_ONE) return kPushAdd;
    if (SR == GBK_LOR_LAND || SR == GBK_STRUCTURAL_BOOL || SR == GBK_CUSTOM_LESS_PLUS) return kPushOne;
    return SR == GBK_FIRST_WINS ? kPushNothing : kPushMin;  // first(y, m) == y
}

constexpr int kHeavyRow = 32;  // rows with at least this many entries are cut into pieces
constexpr int kPiece = 128;    // entries per piece

struct PushArgs {
    const int32_t* ptr;
    const int32_t* idx;
    const void* val;
    const int32_t* ids;
    const void* xv;
    int64_t nf;
    void* y;
    const void* mask;  // elements outside it are left alone (NULL: none)
    int mdt, mmode;
    int take;          // frontier entries per warp
    int2* pieces;      // (frontier entry, first entry of the row's piece)
    int32_t* npieces;
    int32_t room;      // pieces that fit; a row that would pass it is pushed where it stands
};

// One push per lane: entry pos of the row, frontier value x.
template <int SR, typename T>
__device__ __forceinline__ void push_edge(const PushArgs& a, bool valid, int64_t pos, T x, int lane) {
    using S = Semiring<SR, T>;
    constexpr unsigned kFull = 0xffffffffu;
    T* y = (T*)a.y;
    int32_t j = -1 - lane;  // a key no other lane has
    if (valid) {
        j = __ldg(a.idx + pos);
        if (a.mask && !mask_selects(a.mask, a.mdt, a.mmode, j)) {
            valid = false;
            j = -1 - lane;
        }
    }
    if constexpr (push_kind<SR>() == kPushOne) {
        if (valid) y[j] = T(1);
    } else {
        T acc = S::identity();
        if (valid) {
            T v = T(0);
            if constexpr (kUsesValues<SR>) v = __ldg((const T*)a.val + pos);
            acc = S::mul(v, x);
        }
        const unsigned peers = __match_any_sync(kFull, j);
        const int rank = __popc(peers & ((1u << lane) - 1u));
        const int gsize = __popc(peers);
        for (int st = 1; st < 32; st <<= 1) {
            if (!__any_sync(kFull, gsize > st)) break;
            const bool more = (rank % (2 * st)) == 0 && rank + st < gsize;
            const int from = more ? nth_set_bit(peers, rank + st) : lane;
            const T o = __shfl_sync(kFull, acc, from);
            if (more) acc = S::add(acc, o);
        }
        if (valid && rank == 0) {
            if constexpr (push_kind<SR>() == kPushAdd) atomicAdd(y + j, acc);
            else atomic_min_val(y + j, S::add(Lim<T>::max(), acc));
        }
    }
}

// Rows under kHeavyRow entries, edge by edge over the warp's lanes; longer
// ones are listed for k_push_pieces.  Every loop is warp-uniform.
template <int SR, typename T>
__global__ void __launch_bounds__(kPushThreads) k_push(PushArgs a) {
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t ngroups = (a.nf + a.take - 1) / a.take;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; g < ngroups; g += nwarps) {
        const int64_t k = g * a.take + lane;
        int32_t beg = 0, deg = 0;
        T x = T(0);
        if (lane < a.take && k < a.nf) {
            const int32_t u = __ldg(a.ids + k);
            beg = __ldg(a.ptr + u);
            deg = __ldg(a.ptr + u + 1) - beg;
            if constexpr (push_kind<SR>() != kPushOne) x = __ldg((const T*)a.xv + k);
        }
        bool heavy = deg >= kHeavyRow;
        if (heavy) {
            const int32_t np = pieces_of(deg, kPiece);
            const int32_t at = atomicAdd(a.npieces, np);
            if (at >= 0 && at <= a.room - np)
                for (int32_t i = 0; i < np; ++i) a.pieces[at + i] = make_int2((int32_t)k, beg + i * kPiece);
            else if (at >= 0 && at < a.room)
                for (int32_t i = at; i < a.room; ++i) a.pieces[i] = make_int2(-1, 0);
            // what does not fit is pushed here
            heavy = at >= 0 && at <= a.room - np;
        }
        const int32_t dl = heavy ? 0 : deg;
        unsigned lone = __ballot_sync(kFull, dl >= kHeavyRow);
        const int32_t mine = dl >= kHeavyRow ? 0 : dl;
        int32_t incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t up = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += up;
        }
        const int32_t before = incl - mine;
        const int32_t total = __shfl_sync(kFull, incl, 31);
        for (int32_t t0 = 0; t0 < total; t0 += 32) {
            const int32_t t = t0 + lane;
            // the row of edge t: the first lane whose inclusive count exceeds t
            int j = 0;
#pragma unroll
            for (int st = 16; st; st >>= 1)
                if (__shfl_sync(kFull, incl, j + st - 1) <= t) j += st;
            j = min(j, 31);  // lanes past the end
            const int32_t eb = __shfl_sync(kFull, beg, j), ex = __shfl_sync(kFull, before, j);
            const T xj = __shfl_sync(kFull, x, j);
            push_edge<SR, T>(a, t < total, (int64_t)eb + (t - ex), xj, lane);
        }
        while (lone) {  // rows whose pieces did not fit
            const int j = __ffs(lone) - 1;
            lone &= lone - 1;
            const int32_t eb = __shfl_sync(kFull, beg, j), d = __shfl_sync(kFull, deg, j);
            const T xj = __shfl_sync(kFull, x, j);
            for (uint32_t t0 = 0; t0 < (uint32_t)d; t0 += 32)
                push_edge<SR, T>(a, t0 + lane < (uint32_t)d, (int64_t)eb + t0 + lane, xj, lane);
        }
    }
}

// The listed pieces, one warp each.
template <int SR, typename T>
__global__ void __launch_bounds__(kPushThreads) k_push_pieces(PushArgs a) {
    const int lane = threadIdx.x & 31;
    const int32_t listed = *a.npieces;
    const int64_t np = listed < 0 || listed > a.room ? a.room : listed;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t c = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; c < np; c += nwarps) {
        const int2 pc = a.pieces[c];
        if (pc.x < 0) continue;
        T x = T(0);
        if constexpr (push_kind<SR>() != kPushOne) x = __ldg((const T*)a.xv + pc.x);
        const uint32_t end = piece_end(pc.y, kPiece, __ldg(a.ptr + __ldg(a.ids + pc.x) + 1));
#pragma unroll 4
        for (uint32_t e0 = pc.y; e0 < end; e0 += 32) push_edge<SR, T>(a, e0 + lane < end, (int64_t)e0 + lane, x, lane);
    }
}

// y = the identity, 0 outside the mask (if any); the old values are kept in
// `old` (if any) for an accumulator.
template <typename T>
__global__ void k_push_begin(T* y, int64_t n, T ident, T* old, const void* m, int mdt, int mmode, int32_t* npieces) {
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (tid == 0) *npieces = 0;
    for (int64_t i = tid; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (old) old[i] = y[i];
        y[i] = !m || mask_selects(m, mdt, mmode, i) ? ident : T(0);
    }
}

// apply_mask (spmspv.h:17-99), dense form (sparse complements are expanded first)
template <typename T>
__global__ void k_apply_mask_dense(T* y, const T* old, int64_t n, int accum, const void* m, int mdt, int mmode) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        bool sel = mask_selects(m, mdt, mmode, i);
        y[i] = sel ? binop<T>(accum, old[i], y[i]) : T(0);
    }
}

template <typename T>
__global__ void k_apply_mask_ids(T* y, const T* old, const int32_t* ids, int64_t nv, int accum) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nv; k += (int64_t)gridDim.x * blockDim.x) {
        int32_t i = ids[k];
        y[i] = binop<T>(accum, old[i], y[i]);
    }
}

__global__ void k_mark(const int32_t* ids, int64_t nv, uint8_t* flag) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nv; k += (int64_t)gridDim.x * blockDim.x)
        flag[ids[k]] = 1;
}

// One warp per listed row (SpMV_sparse without complement).
template <int SR, typename T>
__global__ void k_spmv_rows(const int32_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                            const T* __restrict__ val, const int32_t* __restrict__ rows, int64_t nr,
                            const T* __restrict__ x, T* __restrict__ y, int accum) {
    using S = Semiring<SR, T>;
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t k = warp; k < nr; k += nwarps) {
        const int32_t r = rows[k];
        T acc = S::identity();
        if constexpr (Semiring<SR, T>::assoc) {
            for (int e = ptr[r] + lane; e < ptr[r + 1]; e += 32) acc = S::add(acc, S::mul(val[e], x[idx[e]]));
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) acc = S::add(acc, __shfl_down_sync(0xffffffffu, acc, off));
        } else {
            if (lane == 0)
                for (int e = ptr[r]; e < ptr[r + 1]; e++) acc = S::add(acc, S::mul(val[e], x[idx[e]]));
        }
        if (lane == 0) y[r] = (accum == GBK_OP_SECOND) ? acc : binop<T>(accum, y[r], acc);
    }
}

inline unsigned grid_cap(int64_t work, int threads) {
    int64_t b = (work + threads - 1) / threads;
    int64_t cap = (int64_t)num_sms() * 8;
    if (b > cap) b = cap;
    return (unsigned)(b > 0 ? b : 1);
}

template <typename T>
int spmspv_t(int sr, const CsrView& v, int accum, const int32_t* ids, const void* xv, int64_t nf, T* y,
             const gbk_mask* mask, cudaStream_t s) {
    const int64_t n = v.nrows == v.ncols ? v.ncols : v.ncols;  // y is indexed by the pushed-to side
    T ident;
    switch (sr) {
        case GBK_MIN_PLUS:
        case GBK_CUSTOM_LESS_PLUS:
        case GBK_MIN_SECOND:
        case GBK_MIN_NOTEQ:
            ident = Lim<T>::max();
            break;
        default:
            ident = T(0);
    }
    // Without an accumulator (second) the mask needs no old values and no pass
    // of its own: elements outside it are set to 0 at the start and never
    // pushed to (a list of ids that is not complemented changes nothing).  A
    // mask that shares memory with y is applied at the end, to the new values.
    const bool apart = !mask || !mask->dense || (const char*)mask->dense >= (const char*)(y + n) ||
                       (const char*)mask->dense + dtype_size(mask->dtype) * (size_t)n <= (const char*)y;
    const bool second = accum == GBK_OP_SECOND && apart;
    if (second && mask && !mask->dense && mask->mode != GBK_MASK_STR_COMP) mask = nullptr;
    // pieces of a frontier without repeats; a small frontier over a huge matrix
    // gets room for its likely ones, and none at all when memory is short
    int64_t room = nf > 0 ? std::min<int64_t>(v.nnz / kHeavyRow + 1, (1 << 20) + 64 * nf) : 0;
    StreamScratch dev(s);
    PushArgs a{v.ptr, v.idx, v.val, ids, xv, nf, y, nullptr, 0, 0, 0, nullptr, nullptr, 0};
    T* old = nullptr;
    uint8_t* flag = nullptr;
    int32_t* mem = nullptr;
    if (dev.get(&mem, 16 + sizeof(int2) * (size_t)room)) room = 0;
    if ((room == 0 && !mem && dev.get(&mem, 16)) || (mask && !second && dev.get(&old, sizeof(T) * (size_t)n)) ||
        (mask && !mask->dense && mask->mode == GBK_MASK_STR_COMP && dev.get(&flag, (size_t)n))) {
        set_error("gbk_spmspv: out of device memory");
        return GBK_OUT_OF_MEMORY;
    }
    a.npieces = mem;
    a.pieces = (int2*)(mem + 4);
    a.room = (int32_t)room;
    // a small frontier gets more warps: 8 entries each until they fill the SMs
    a.take = nf < (int64_t)num_sms() * 64 * 32 ? 8 : 32;
    if (flag) {
        GBK_CUDA(cudaMemsetAsync(flag, 0, n, s));
        if (mask->nvals > 0) {
            k_mark<<<grid_cap(mask->nvals, 256), 256, 0, s>>>(mask->ids, mask->nvals, flag);
            GBK_LAUNCHED();
        }
    }
    const void* dmask = !mask ? nullptr : mask->dense ? mask->dense : flag;
    const int mdt = mask && mask->dense ? mask->dtype : GBK_BOOL, mmode = mask ? mask->mode : 0;
    if (second) {
        a.mask = dmask;
        a.mdt = mdt;
        a.mmode = mmode;
    }
    if (n > 0) {
        k_push_begin<T><<<grid_cap(n, 256), 256, 0, s>>>(y, n, ident, old, a.mask, a.mdt, a.mmode, a.npieces);
        GBK_LAUNCHED();
    }
    if (nf > 0 && n > 0) {
        const unsigned grid = grid_cap((nf + a.take - 1) / a.take * 32, kPushThreads);
        const unsigned pgrid = grid_cap(room * 32, kPushThreads);
#define PUSH_CASE(SRV)                                                 \
    case SRV:                                                          \
        if constexpr (push_kind<SRV>() != kPushNothing) {              \
            k_push<SRV, T><<<grid, kPushThreads, 0, s>>>(a);           \
            GBK_LAUNCHED();                                            \
            k_push_pieces<SRV, T><<<pgrid, kPushThreads, 0, s>>>(a);   \
            GBK_LAUNCHED();                                            \
        }                                                              \
        break;
        switch (sr) {
            PUSH_CASE(GBK_PLUS_TIMES)
            PUSH_CASE(GBK_LOR_LAND)
            PUSH_CASE(GBK_FIRST_WINS)
            PUSH_CASE(GBK_FIRST_MIN)
            PUSH_CASE(GBK_PLUS_SECOND)
            PUSH_CASE(GBK_STRUCTURAL_BOOL)
            PUSH_CASE(GBK_MIN_PLUS)
            PUSH_CASE(GBK_CUSTOM_LESS_PLUS)
            PUSH_CASE(GBK_MIN_SECOND)
            PUSH_CASE(GBK_MIN_NOTEQ)
            PUSH_CASE(GBK_PLUS_ONE)
            default:
                set_error("gbk_spmspv: unknown semiring %d", sr);
                return GBK_INVALID_VALUE;
        }
#undef PUSH_CASE
    }
    if (mask && !second && n > 0) {
        if (dmask) {
            k_apply_mask_dense<T><<<grid_cap(n, 256), 256, 0, s>>>(y, old, n, accum, dmask, mdt, mmode);
            GBK_LAUNCHED();
        } else if (mask->nvals > 0) {
            k_apply_mask_ids<T><<<grid_cap(mask->nvals, 256), 256, 0, s>>>(y, old, mask->ids, mask->nvals, accum);
            GBK_LAUNCHED();
        }
    }
    return GBK_SUCCESS;
}

template <typename T>
int rows_t(int sr, const CsrView& v, int accum, const T* x, T* y, const int32_t* rows, int64_t nr, cudaStream_t s) {
    if (nr == 0) return GBK_SUCCESS;
    const unsigned grid = grid_cap(nr * 32, 256);
#define ROWS_CASE(SRV)                                                                                    \
    case SRV:                                                                                             \
        k_spmv_rows<SRV, T><<<grid, 256, 0, s>>>(v.ptr, v.idx, (const T*)v.val, rows, nr, x, y, accum); \
        break;
    switch (sr) {
        ROWS_CASE(GBK_PLUS_TIMES)
        ROWS_CASE(GBK_LOR_LAND)
        ROWS_CASE(GBK_FIRST_WINS)
        ROWS_CASE(GBK_FIRST_MIN)
        ROWS_CASE(GBK_PLUS_SECOND)
        ROWS_CASE(GBK_STRUCTURAL_BOOL)
        ROWS_CASE(GBK_MIN_PLUS)
        ROWS_CASE(GBK_CUSTOM_LESS_PLUS)
        ROWS_CASE(GBK_MIN_SECOND)
        ROWS_CASE(GBK_MIN_NOTEQ)
        ROWS_CASE(GBK_PLUS_ONE)
        default:
            set_error("unknown semiring %d", sr);
            return GBK_INVALID_VALUE;
    }
#undef ROWS_CASE
    GBK_LAUNCHED();
    return GBK_SUCCESS;
}

}  // namespace

}  // namespace gbk

using namespace gbk;

extern "C" {

int gbk_spmspv(gbk_matrix A, int transpose, gbk_semiring sr, gbk_binop accum, gbk_dtype dtype,
               const int32_t* x_ids, const void* x_vals, int64_t x_nvals, void* y, const gbk_mask* mask,
               void* stream) {
    GBK_REQUIRE(A && y, GBK_NULL_POINTER, "gbk_spmspv: NULL argument");
    GBK_REQUIRE(x_nvals == 0 || (x_ids && x_vals), GBK_NULL_POINTER, "gbk_spmspv: NULL frontier");
    GBK_REQUIRE(dtype == A->vtype, GBK_DOMAIN_MISMATCH, "gbk_spmspv: vector type %d != matrix type %d", (int)dtype,
                (int)A->vtype);
    cudaStream_t s = (cudaStream_t)stream;
    // mxv pushes along columns of A (the CSC), vxm along rows (the CSR): spmspv.h:125-146
    if (!transpose) {
        int rc = ensure_csc(A, s);
        if (rc) return rc;
    }
    const CsrView& v = transpose ? A->csr : A->csc;
    if (dtype == GBK_F32) return spmspv_t<float>(sr, v, accum, x_ids, x_vals, x_nvals, (float*)y, mask, s);
    if (dtype == GBK_I32) return spmspv_t<int32_t>(sr, v, accum, x_ids, x_vals, x_nvals, (int32_t*)y, mask, s);
    set_error("gbk_spmspv: element type %d unsupported", (int)dtype);
    return GBK_UNSUPPORTED;
}

int gbk_mxv_sparse_mask(gbk_matrix A, int transpose, gbk_semiring sr, gbk_binop accum, gbk_dtype dtype,
                        const void* x, void* y, const int32_t* mask_ids, int64_t mask_nvals, gbk_mask_mode mask_mode,
                        void* stream) {
    GBK_REQUIRE(A && x && y, GBK_NULL_POINTER, "gbk_mxv_sparse_mask: NULL argument");
    GBK_REQUIRE(mask_nvals == 0 || mask_ids, GBK_NULL_POINTER, "gbk_mxv_sparse_mask: NULL mask ids");
    GBK_REQUIRE(dtype == A->vtype, GBK_DOMAIN_MISMATCH, "gbk_mxv_sparse_mask: type mismatch");
    cudaStream_t s = (cudaStream_t)stream;
    if (transpose) {
        int rc = ensure_csc(A, s);
        if (rc) return rc;
    }
    const CsrView& v = transpose ? A->csc : A->csr;
    if (mask_mode == GBK_MASK_STR_COMP) {  // spmv_csr.h:218-255: densify, complement
        uint8_t* flag = nullptr;
        const int64_t n = v.nrows;
        GBK_CUDA(cudaMallocAsync((void**)&flag, n > 0 ? n : 1, s));
        GBK_CUDA(cudaMemsetAsync(flag, 0, n > 0 ? n : 1, s));
        if (mask_nvals > 0) {
            k_mark<<<grid_cap(mask_nvals, 256), 256, 0, s>>>(mask_ids, mask_nvals, flag);
            GBK_LAUNCHED();
        }
        int rc = spmv_csr(v, sr, accum, dtype, x, y, flag, GBK_BOOL, GBK_MASK_STR_COMP, s);
        cudaFreeAsync(flag, s);
        return rc;
    }
    if (dtype == GBK_F32) return rows_t<float>(sr, v, accum, (const float*)x, (float*)y, mask_ids, mask_nvals, s);
    if (dtype == GBK_I32)
        return rows_t<int32_t>(sr, v, accum, (const int32_t*)x, (int32_t*)y, mask_ids, mask_nvals, s);
    set_error("gbk_mxv_sparse_mask: element type %d unsupported", (int)dtype);
    return GBK_UNSUPPORTED;
}

}  // extern "C"
