// Unmasked SpGEMM C = A (+.x) B in column windows: one warp (for many products a
// CTA) per (row of C, window of 1,280 or 2,048 columns), the window's sums in shared
// memory.
//
// The warp walks the entries A_ik of its row in order; of every row k of B it
// takes the part inside its window (the parts' bounds are tabulated per call)
// and adds A_ik * B_kj to the sum of column j, 32 entries of B a step.  A row
// of B holds a column once, so the lanes of a step never meet in a sum and the
// updates are plain shared-memory loads and stores; a column's sum is formed
// in the order of A's entries, whatever the schedule, so results repeat bit
// for bit.  The window is then scanned in column order, which leaves the rows
// column-sorted without sorting anything.  Replaces SpMSpM_unmasked_ikj
// (src/backend/spmspm/spmspm_hash_based_gustavson.h:9-148, a hash map per row
// of C); sums equal to 0 are dropped as the reference keeps only val != 0.
//
// B's rows must be column-sorted without repeats and B not too wide for the
// number of products (window_pays); mxm_window reports anything else as not
// done and the caller expands and sorts the products.
//
// A A of an undirected R-MAT graph of 2^14 vertices, 157 M products, 46 M
// entries: 1.3 ms a call, where it took 11.7 ms by expansion and sorting, which
// move every product through memory several times; what is left is the sums
// (0.82 ms) and the result's move to its place (0.24 ms).  2^15, 445 M products,
// in two blocks: 4.5 ms, 29 by expansion.
#include <cub/cub.cuh>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "internal.h"

namespace gbk {

namespace {

constexpr int64_t kMaxColumns = 131072;  // of B
constexpr unsigned kAll = 0xffffffffu;

// Semirings whose identity may also be a sum (min over values that reach the
// largest one) keep a flag per column; for the others the identity is 0, which
// is dropped, so an untouched column needs no flag.
template <int SR>
constexpr bool flagged() {
    return SR == GBK_MIN_PLUS || SR == GBK_MIN_SECOND;
}

// Semirings whose mul reads B_kj.
template <int SR>
constexpr bool kReadsB = SR != GBK_PLUS_ONE;

// Float sums are formed in 64 bits: a column's sum has as many terms as A's row
// has entries at most, and 32-bit sums in order lose more than the expansion's
// (terms of [0, 1): 6.1e-8 from the 64-bit sums at 16 terms, 7.9e-7 at 4,000;
// 5.2e-8 and 5.4e-8 by expansion).  Their windows are narrower, so that 21 warps
// fit an SM.  A A in ms, R-MAT 2^14 | 2^15 | 2^12 | uniform 2^14, 16 entries a row:
// 1,280 columns, 3 warps a CTA 1.32 | 4.5 | 0.32 | 0.71; 1,024 columns (27 warps)
// 1.36 | 4.7 | 0.33 | 0.71; 2,048 (12 warps) 1.66 | 5.6 | 0.31 | 0.89; 7 warps a CTA
// 1.47 | 4.9 | 0.34 | 0.72; 32-bit sums, 2,048 columns, 24 warps 1.37 | 4.8 | 0.30 | 0.58.
template <int SR, typename T>
struct Shape {
    static constexpr bool kWide = std::is_same<T, float>::value &&
                                  (SR == GBK_PLUS_TIMES || SR == GBK_PLUS_SECOND || SR == GBK_PLUS_ONE);
    using Sum = std::conditional_t<kWide, double, T>;
    static constexpr int kCols = kWide ? 1280 : 2048;  // columns per window
    static constexpr int kWarps = kWide ? 3 : 8;       // per CTA
    static constexpr int kSteps = kWide ? 6 : 8;       // 32-entry steps of B a warp loads before it adds the first
    static constexpr int kCtas = kWide ? 7 : flagged<SR>() ? 2 : 3;  // on an SM
    static constexpr int kSmem = (int)(sizeof(Sum) + (flagged<SR>() ? 1 : 0)) * kCols * kWarps;
};

constexpr int kHeavyClass = 31 - 12;  // tasks of 2^12 products or more are worked on by a whole CTA

struct WindowHead {
    unsigned long long products;
    unsigned long long drops;       // entries of B not above the one before them
    unsigned long long row_drops;   // those of them that start a row
    unsigned long long pad;
};

template <int N>
__device__ __forceinline__ void block_add(const unsigned long long (&x)[N], unsigned long long* out) {
    __shared__ unsigned long long part[N][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        unsigned long long v = x[k];
#pragma unroll
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(kAll, v, o);
        if (lane == 0) part[k][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x < N) {
        unsigned long long v = 0;
        for (int w = 0; w < nw; ++w) v += part[threadIdx.x][w];
        if (v) atomicAdd(out + threadIdx.x, v);
    }
}

// Products of A B, and whether B's rows are strictly ascending (they are when
// every descent starts a row).
__global__ void __launch_bounds__(256) k_win_head(const int32_t* __restrict__ aidx, int64_t annz,
                                                  const int32_t* __restrict__ bptr, const int32_t* __restrict__ bidx,
                                                  int64_t bn, int64_t bnnz, WindowHead* head) {
    unsigned long long x[3] = {0, 0, 0};
    const int64_t nth = (int64_t)gridDim.x * blockDim.x, tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t e = tid; e < annz; e += nth) {
        const int32_t k = aidx[e];
        x[0] += bptr[k + 1] - bptr[k];
    }
    for (int64_t e = tid + 1; e < bnnz; e += nth) x[1] += bidx[e] <= bidx[e - 1];
    for (int64_t r = tid; r < bn; r += nth) {
        const int32_t b = bptr[r];
        if (b > 0 && bptr[r + 1] > b) x[2] += bidx[b] <= bidx[b - 1];
    }
    block_add(x, &head->products);
}

// seg[k * (nw + 1) + w]: first entry of B's row k in window w or later.
__global__ void __launch_bounds__(256) k_win_bounds(const int32_t* __restrict__ bptr, const int32_t* __restrict__ bidx,
                                                    int64_t total, int nw, int cols, int32_t* __restrict__ seg) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int64_t k = i / (nw + 1);
    const int w = (int)(i - k * (nw + 1));
    int32_t lo = bptr[k], hi = bptr[k + 1];
    const int32_t col = w * cols;  // at most kMaxColumns and a window
    if (w == 0) hi = lo;
    if (w == nw) lo = hi;
    while (lo < hi) {
        const int32_t mid = lo + ((hi - lo) >> 1);
        if (bidx[mid] < col)
            lo = mid + 1;
        else
            hi = mid;
    }
    seg[i] = lo;
}

constexpr int kClasses = 32;

__device__ __forceinline__ int task_class(long long products) {  // heaviest first
    return 31 - min(31, 63 - __clzll(products));
}

// Per task (row, window): its products, bounded by the window's columns
// (room[task]; room[ntasks] = 0), and the number of tasks per class.
__global__ void __launch_bounds__(256) k_win_tasks(const int32_t* __restrict__ aptr, const int32_t* __restrict__ aidx,
                                                   const int32_t* __restrict__ seg, int64_t ntasks, int nw, int cols, int64_t m,
                                                   int64_t* __restrict__ room, uint8_t* __restrict__ cls,
                                                   int32_t* __restrict__ hist) {
    __shared__ int32_t h[kClasses];
    if (threadIdx.x < kClasses) h[threadIdx.x] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < ntasks; t += nwarps) {
        const int32_t row = (int32_t)t / nw, w = (int32_t)t - row * nw;  // tasks are int32
        long long sum = 0;
        const uint32_t a1 = aptr[row + 1];
        for (uint32_t e = aptr[row] + lane; e < a1; e += 32) {
            const int32_t* s = seg + (int64_t)aidx[e] * (nw + 1) + w;
            sum += s[1] - s[0];
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(kAll, sum, o);
        if (lane == 0) {
            const long long width = m - (int64_t)w * cols < cols ? m - (int64_t)w * cols : cols;
            room[t] = sum < width ? sum : width;
            const int c = sum > 0 ? task_class(sum) : 255;
            cls[t] = (uint8_t)c;
            if (sum > 0) atomicAdd(h + c, 1);
            if (t == 0) room[ntasks] = 0;
        }
    }
    __syncthreads();
    if (threadIdx.x < kClasses && h[threadIdx.x]) atomicAdd(hist + threadIdx.x, h[threadIdx.x]);
}

// Number of tasks per class of a block's tasks.
__global__ void __launch_bounds__(256) k_win_classes(const uint8_t* __restrict__ cls, int64_t ntasks,
                                                     int32_t* __restrict__ hist) {
    __shared__ int32_t h[kClasses];
    if (threadIdx.x < kClasses) h[threadIdx.x] = 0;
    __syncthreads();
    const int64_t nth = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < ntasks; t += nth)
        if (cls[t] != 255) atomicAdd(h + cls[t], 1);
    __syncthreads();
    if (threadIdx.x < kClasses && h[threadIdx.x]) atomicAdd(hist + threadIdx.x, h[threadIdx.x]);
}

// The tasks [task0, task0 + ntasks) with products, heaviest class first (inside
// a class in any order); cls and order from task0 on.
__global__ void __launch_bounds__(256) k_win_order(const uint8_t* __restrict__ cls, int64_t task0, int64_t ntasks,
                                                   const int32_t* __restrict__ hist, int32_t* __restrict__ cursor,
                                                   int32_t* __restrict__ order) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int c = t < ntasks ? cls[t] : 255;
    const int lane = threadIdx.x & 31;
    const unsigned peers = __match_any_sync(kAll, c);
    if (c == 255) return;
    int32_t at = 0;
    const int lead = __ffs(peers) - 1;
    if (lane == lead) {
        for (int k = 0; k < c; ++k) at += hist[k];
        at += atomicAdd(cursor + c, __popc(peers));
    }
    at = __shfl_sync(peers, at, lead);
    order[at + __popc(peers & ((1u << lane) - 1u))] = (int32_t)(task0 + t);
}

struct WindowArgs {
    const int32_t* aptr;
    const int32_t* aidx;
    const void* aval;
    const int32_t* bidx;
    const void* bval;
    const int32_t* seg;
    int nw;
    int64_t task0;            // first task of the block
    const int32_t* order;     // tasks to run
    int64_t nheavy;           // the first ones, a CTA each
    int64_t ntasks;           // their number
    const int64_t* off;       // room before each task
    int64_t off0;             // room before the block
    int32_t* tcol;            // the tasks' entries, each task's at off[task] - off0
    void* tval;
    int64_t* count;           // entries of each task (relative to task0)
    unsigned long long* next; // the next heavy task, the next other one
};

// A warp's sums of one window over the entries [a0, a1) of a row of A.
template <int SR, typename T>
__device__ __forceinline__ void window_sums(const WindowArgs& g, int w, uint32_t a0, uint32_t a1,
                                            typename Shape<SR, T>::Sum* acc, uint8_t* seen, int lane) {
    using S = Semiring<SR, T>;
    using Sum = typename Shape<SR, T>::Sum;
    constexpr int kSteps = Shape<SR, T>::kSteps;
    const T* __restrict__ aval = (const T*)g.aval;
    const T* __restrict__ bval = (const T*)g.bval;
    const int32_t* __restrict__ bidx = g.bidx;
    const int32_t col0 = w * Shape<SR, T>::kCols;
    const int32_t* __restrict__ seg = g.seg + w;
    for (; a0 < a1; a0 += 32) {
        uint32_t sb = 0, se = 0;
        T av = T(0);
        if (a0 + lane < a1) {
            const int32_t k = g.aidx[a0 + lane];
            av = aval[a0 + lane];
            sb = __ldg(seg + (int64_t)k * (g.nw + 1));
            se = __ldg(seg + (int64_t)k * (g.nw + 1) + 1);
        }
        unsigned todo = __ballot_sync(kAll, se > sb);
        uint32_t p = 0, e = 0;  // what is left of the current part of a row of B
        T a = T(0);
        while (todo || p < e) {
            int32_t c[kSteps];
            T b[kSteps], f[kSteps];
#pragma unroll
            for (int u = 0; u < kSteps; ++u) {
                if (p >= e && todo) {
                    const int j = __ffs(todo) - 1;
                    todo &= todo - 1;
                    p = __shfl_sync(kAll, sb, j);
                    e = __shfl_sync(kAll, se, j);
                    a = __shfl_sync(kAll, av, j);
                }
                const bool live = p + lane < e;
                c[u] = live ? __ldg(bidx + p + lane) : -1;
                b[u] = live && kReadsB<SR> ? __ldg(bval + p + lane) : T(0);
                f[u] = a;
                p += 32;
            }
#pragma unroll
            for (int u = 0; u < kSteps; ++u) {
                if (c[u] >= 0) {
                    const int q = c[u] - col0;
                    const T x = S::mul(f[u], b[u]);
                    if constexpr (flagged<SR>()) {
                        acc[q] = seen[q] ? S::add(acc[q], x) : x;
                        seen[q] = 1;
                    } else if constexpr (std::is_same<Sum, T>::value) {
                        acc[q] = S::add(acc[q], x);
                    } else {
                        acc[q] += (Sum)x;
                    }
                }
                __syncwarp();  // the next step may meet the same columns in other lanes
            }
        }
    }
}

// The window's sums in column order to the task's room, cleared behind the scan.
template <int SR, typename T>
__device__ __forceinline__ void window_out(const WindowArgs& g, int64_t task, int w, typename Shape<SR, T>::Sum* acc,
                                           uint8_t* seen, int lane) {
    int64_t at = g.off[task] - g.off0;
    const int64_t first = at;
    T* tval = (T*)g.tval;
    constexpr int kAhead = 4;  // loads in flight
    static_assert(Shape<SR, T>::kCols % (32 * kAhead) == 0, "the scan takes 128 columns at a time");
    for (int q0 = lane; q0 < Shape<SR, T>::kCols; q0 += 32 * kAhead) {
        T v[kAhead];
        bool keep[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            v[k] = (T)acc[q0 + 32 * k];
            keep[k] = v[k] != T(0);
            if constexpr (flagged<SR>()) keep[k] = keep[k] && seen[q0 + 32 * k];
        }
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            const int q = q0 + 32 * k;
            if constexpr (flagged<SR>()) seen[q] = 0;
            acc[q] = Semiring<SR, T>::identity();
            const unsigned bal = __ballot_sync(kAll, keep[k]);
            if (!bal) continue;
            if (keep[k]) {
                const int64_t o = at + __popc(bal & ((1u << lane) - 1u));
                g.tcol[o] = w * Shape<SR, T>::kCols + q;
                tval[o] = v[k];
            }
            at += __popc(bal);
        }
    }
    __syncwarp();
    if (lane == 0) g.count[task - g.task0] = at - first;
}

// Bound by the steps (a 32-entry piece of a row of B: two coalesced loads, a
// shared-memory load, add and store), about 30 instructions each; kSteps of
// them are loaded ahead, across the ends of B's rows, to cover L2's latency.
// A heavy task is worked on by a whole CTA: its warps take the row's entries
// 32 at a time in turn, each into a window of its own, and at the end each
// thread adds up the sums of its columns in the order of the warps.
template <int SR, typename T>
__global__ void __launch_bounds__(32 * Shape<SR, T>::kWarps, Shape<SR, T>::kCtas) k_win_numeric(WindowArgs g) {
    using S = Semiring<SR, T>;
    using Sum = typename Shape<SR, T>::Sum;
    constexpr int kCols = Shape<SR, T>::kCols, kWarps = Shape<SR, T>::kWarps;
    extern __shared__ uint8_t smem[];
    __shared__ unsigned long long s_next;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Sum* const all = (Sum*)smem;
    uint8_t* const all_seen = smem + sizeof(Sum) * kCols * kWarps;  // flagged semirings only
    Sum* acc = all + warp * kCols;
    uint8_t* seen = all_seen + warp * kCols;
    for (int i = lane; i < kCols; i += 32) {
        acc[i] = S::identity();
        if constexpr (flagged<SR>()) seen[i] = 0;
    }
    __syncwarp();
    if (g.nheavy > 0) {
        for (;;) {
            __syncthreads();  // warp 0 has written the last task's sums
            if (threadIdx.x == 0) s_next = atomicAdd(g.next, 1ull);
            __syncthreads();
            if ((long long)s_next >= g.nheavy) break;
            const int32_t task = g.order[s_next];
            const int32_t row = task / g.nw, w = task - row * g.nw;
            const int32_t a0 = g.aptr[row], a1 = g.aptr[row + 1];
            const int32_t per = min(32, pieces_of(a1 - a0, kWarps));  // entries of A per warp and turn
            for (int64_t from = (int64_t)a0 + warp * per; from < a1; from += kWarps * per)
                window_sums<SR, T>(g, w, (uint32_t)from, (uint32_t)(from + per < a1 ? from + per : a1), acc, seen, lane);
            __syncthreads();
            for (int q = threadIdx.x; q < kCols; q += 32 * kWarps) {
                Sum tot = S::identity();
                bool any = false;
#pragma unroll
                for (int i = 0; i < kWarps; ++i) {
                    const Sum part = all[i * kCols + q];
                    all[i * kCols + q] = S::identity();
                    if constexpr (flagged<SR>()) {
                        if (!all_seen[i * kCols + q]) continue;
                        all_seen[i * kCols + q] = 0;
                        tot = any ? S::add(tot, part) : part;
                        any = true;
                    } else if constexpr (std::is_same<Sum, T>::value) {
                        tot = S::add(tot, part);
                    } else {
                        tot += part;
                    }
                }
                all[q] = tot;
                if constexpr (flagged<SR>()) all_seen[q] = any;
            }
            __syncthreads();
            if (warp == 0) window_out<SR, T>(g, task, w, acc, seen, lane);
        }
    }
    for (;;) {
        unsigned long long i = 0;
        if (lane == 0) i = atomicAdd(g.next + 1, 1ull);
        i = __shfl_sync(kAll, i, 0) + g.nheavy;
        if ((long long)i >= g.ntasks) break;
        const int32_t task = g.order[i];
        const int32_t row = task / g.nw, w = task - row * g.nw;
        window_sums<SR, T>(g, w, g.aptr[row], g.aptr[row + 1], acc, seen, lane);
        __syncwarp();
        window_out<SR, T>(g, task, w, acc, seen, lane);
    }
}

// Task t's entries from its room to their place (fin: entries before each task).
__global__ void __launch_bounds__(256) k_win_gather(int64_t task0, int64_t ntasks, const int64_t* __restrict__ off,
                                                    int64_t off0, const int64_t* __restrict__ fin,
                                                    const int32_t* __restrict__ tcol, const uint32_t* __restrict__ tval,
                                                    int32_t* __restrict__ col, uint32_t* __restrict__ val) {
    const int lane = threadIdx.x & 31;
    const int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= ntasks) return;
    const int64_t b = fin[t], n = fin[t + 1] - b, from = off[task0 + t] - off0;
    for (int64_t i = lane; i < n; i += 32) {
        col[b + i] = __ldcs(tcol + from + i);
        val[b + i] = __ldcs(tval + from + i);
    }
}

// Row starts of the block's rows, after `base` entries; the last block also writes the end.
__global__ void k_win_ptr(const int64_t* __restrict__ fin, int64_t row0, int64_t nrows, int nw, int64_t base,
                          int32_t* __restrict__ ptr) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r <= nrows) ptr[row0 + r] = (int32_t)(base + fin[r * nw]);
}

__global__ void k_win_row_room(const int64_t* __restrict__ off, int64_t nrows, int nw, int64_t* __restrict__ roff) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r <= nrows) roff[r] = off[r * nw];
}

unsigned nb(int64_t n) { return (unsigned)std::max<int64_t>(1, (n + 255) / 256); }

// ptr, col and val of C, freed unless handed over.
struct Owned {
    cudaStream_t s;
    void* p[3] = {nullptr, nullptr, nullptr};
    explicit Owned(cudaStream_t st) : s(st) {}
    Owned(const Owned&) = delete;
    ~Owned() {
        for (void* q : p)
            if (q) cudaFreeAsync(q, s);
    }
    int get(int k, size_t bytes) {
        const int rc = result_alloc(&p[k], bytes, s);
        if (rc == GBK_OUT_OF_MEMORY) set_error("gbk_mxm: out of device memory for the result");
        return rc;
    }
    int get_entries(size_t entries, size_t elem) {
        const int rc = get(1, 4 * entries);
        return rc ? rc : get(2, elem * entries);
    }
};

// Windows or expansion, by their times in ns.  A (row, window) task costs 0.5,
// mostly the scan of its columns, and an (entry of A, window) pair 0.2; integer
// sums and or-and about 0.7 of that.  The expansion costs 0.085 a product and is
// 0.15 ms slower to start, 0.85 ms where the sort takes several passes.  ms by
// windows | by expansion, float sums, both close to the line: uniform graphs of
// 2^15 vertices with 4, 16 and 32 entries a row 0.89 | 1.2, 2.0 | 1.75 and
// 3.6 | 3.8, undirected R-MAT 2^16 with edge factors 1 and 2 2.0 | 1.9 and
// 3.0 | 3.7.  Far from it: uniform 2^17, 16 a row, 24 | 5.2; R-MAT 2^16, edge
// factor 4, 4.7 | 10.
// The table of B's parts must not outgrow what the expansion would hold (a
// hypersparse B has far more rows than products).  Windows counted as 2,048
// columns each.
bool window_pays(const CsrView& a, const CsrView& b, unsigned long long products, bool light) {
    const int64_t nw = (b.ncols + 2047) / 2048;
    const double windows = (light ? 0.7 : 1.0) * (0.5 * (double)a.nrows + 0.2 * (double)a.nnz) * (double)nw;
    const double expansion = 0.085 * (double)products + (products > (1u << 18) ? 0.85e6 : 0.15e6);
    return windows <= expansion && (unsigned long long)b.nrows * (nw + 1) <= 4 * products + 65536;
}

template <int SR, typename T>
int window_t(gbk_matrix* out, const CsrView& a, const CsrView& b, int64_t block_entries, bool* done, cudaStream_t s) {
    const int64_t n = a.nrows, m = b.ncols;
    using Sh = Shape<SR, T>;
    const int nw = (int)((m + Sh::kCols - 1) / Sh::kCols);
    const int64_t ntasks = n * nw;
    if (ntasks >= INT32_MAX) return GBK_SUCCESS;  // tasks are int32
    StreamScratch dev(s);
    WindowHead* d_head = nullptr;
    if (dev.get(&d_head, 512)) return GBK_SUCCESS;  // not done, as for all scratch: the expansion may still fit
    unsigned long long* d_next = (unsigned long long*)d_head + 4;
    int32_t* d_hist = (int32_t*)(d_next + 2);
    int32_t* d_cursor = d_hist + kClasses;
    GBK_CUDA(cudaMemsetAsync(d_head, 0, 512, s));
    k_win_head<<<(unsigned)std::min<int64_t>(nb(std::max(a.nnz, b.nnz)), (int64_t)num_sms() * 8), 256, 0, s>>>(
        a.idx, a.nnz, b.ptr, b.idx, b.nrows, b.nnz, d_head);
    GBK_LAUNCHED();
    WindowHead head;
    GBK_CUDA(cudaMemcpyAsync(&head, d_head, sizeof(head), cudaMemcpyDeviceToHost, s));
    GBK_CUDA(cudaStreamSynchronize(s));
    if (head.drops != head.row_drops || !window_pays(a, b, head.products, !Sh::kWide && !flagged<SR>())) return GBK_SUCCESS;
    // the parts of B's rows and the tasks' room
    int32_t *seg = nullptr, *order = nullptr;
    int64_t *room = nullptr, *off = nullptr;
    uint8_t* cls = nullptr;
    if (dev.get(&seg, 4 * (size_t)b.nrows * (nw + 1)) || dev.get(&order, 4 * (size_t)ntasks) ||
        dev.get(&room, 8 * (size_t)(ntasks + 1)) || dev.get(&off, 8 * (size_t)(ntasks + 1)) ||
        dev.get(&cls, (size_t)ntasks))
        return GBK_SUCCESS;
    k_win_bounds<<<nb(b.nrows * (nw + 1)), 256, 0, s>>>(b.ptr, b.idx, b.nrows * (nw + 1), nw, Sh::kCols, seg);
    GBK_LAUNCHED();
    k_win_tasks<<<(unsigned)std::min<int64_t>((ntasks + 7) / 8, (int64_t)num_sms() * 8), 256, 0, s>>>(
        a.ptr, a.idx, seg, ntasks, nw, Sh::kCols, m, room, cls, d_hist);
    GBK_LAUNCHED();
    k_win_order<<<nb(ntasks), 256, 0, s>>>(cls, 0, ntasks, d_hist, d_cursor, order);
    GBK_LAUNCHED();
    size_t tb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb, room, off, ntasks + 1, s);
    void* tmp = nullptr;
    if (dev.get(&tmp, tb)) return GBK_SUCCESS;
    GBK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, room, off, ntasks + 1, s));
    count_launch(1);
    int64_t total_room = 0;
    std::vector<int32_t> hist(kClasses);  // tasks per class of each block
    GBK_CUDA(cudaMemcpyAsync(&total_room, off + ntasks, 8, cudaMemcpyDeviceToHost, s));
    GBK_CUDA(cudaMemcpyAsync(hist.data(), d_hist, 4 * kClasses, cudaMemcpyDeviceToHost, s));
    GBK_CUDA(cudaStreamSynchronize(s));
    // blocks of whole rows with room for at most block_entries entries (a single row may exceed it)
    std::vector<int64_t> cuts{0, n}, hroff{0, total_room};  // cut rows and the room before them
    if (total_room > block_entries) {
        int64_t* roff = nullptr;
        if (dev.get(&roff, 8 * (size_t)(n + 1))) return GBK_SUCCESS;
        k_win_row_room<<<nb(n + 1), 256, 0, s>>>(off, n, nw, roff);
        GBK_LAUNCHED();
        std::vector<int64_t> all(n + 1);
        GBK_CUDA(cudaMemcpyAsync(all.data(), roff, 8 * (size_t)(n + 1), cudaMemcpyDeviceToHost, s));
        GBK_CUDA(cudaStreamSynchronize(s));
        cuts.assign(1, 0);
        hroff.assign(1, 0);
        while (cuts.back() < n) {
            const int64_t r = cuts.back();
            int64_t r1 = std::upper_bound(all.begin() + r + 1, all.end(), all[r] + block_entries) - all.begin() - 1;
            r1 = std::max(r1, r + 1);
            cuts.push_back(r1);
            hroff.push_back(all[r1]);
        }
    }
    const size_t nblocks = cuts.size() - 1;
    if (nblocks > 1) {  // each block's tasks in an order of their own
        int32_t* d_bhist = nullptr;  // per block: tasks per class, then cursors
        const size_t bytes = 4 * 2 * kClasses * nblocks;
        if (dev.get(&d_bhist, bytes)) return GBK_SUCCESS;
        GBK_CUDA(cudaMemsetAsync(d_bhist, 0, bytes, s));
        for (size_t c = 0; c < nblocks; ++c) {
            const int64_t t0 = cuts[c] * nw, nt = (cuts[c + 1] - cuts[c]) * nw;
            int32_t* h = d_bhist + 2 * kClasses * c;
            k_win_classes<<<(unsigned)std::min<int64_t>(nb(nt), (int64_t)num_sms() * 8), 256, 0, s>>>(cls + t0, nt, h);
            GBK_LAUNCHED();
            k_win_order<<<nb(nt), 256, 0, s>>>(cls + t0, t0, nt, h, h + kClasses, order + t0);
            GBK_LAUNCHED();
        }
        hist.resize(2 * kClasses * nblocks);
        GBK_CUDA(cudaMemcpyAsync(hist.data(), d_bhist, bytes, cudaMemcpyDeviceToHost, s));
        GBK_CUDA(cudaStreamSynchronize(s));
    }
    int64_t max_room = 0;
    for (size_t c = 0; c < nblocks; ++c) max_room = std::max(max_room, hroff[c + 1] - hroff[c]);
    int32_t* tcol = nullptr;
    T* tval = nullptr;
    int64_t* count = room;  // the rooms have been scanned
    int64_t* fin = nullptr;
    if (dev.get(&tcol, 4 * (size_t)max_room) || dev.get(&tval, sizeof(T) * (size_t)max_room) ||
        dev.get(&fin, 8 * (size_t)(ntasks + 1)))
        return GBK_SUCCESS;
    GBK_CUDA(cudaFuncSetAttribute(k_win_numeric<SR, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::kSmem));
    Owned own(s);
    if (const int rc = own.get(0, 4 * (size_t)(n + 1))) return rc;
    std::vector<int32_t*> bcol(nblocks, nullptr);
    std::vector<T*> bval(nblocks, nullptr);
    std::vector<int64_t> bcnt(nblocks, 0);
    int64_t total = 0;
    for (size_t c = 0; c < nblocks; ++c) {
        const int64_t t0 = cuts[c] * nw, nt = (cuts[c + 1] - cuts[c]) * nw;
        int64_t run = 0, nheavy = 0;
        for (int k = 0; k < kClasses; ++k) {
            run += hist[2 * kClasses * c + k];
            if (k <= kHeavyClass) nheavy += hist[2 * kClasses * c + k];
        }
        GBK_CUDA(cudaMemsetAsync(count, 0, 8 * (size_t)(nt + 1), s));
        GBK_CUDA(cudaMemsetAsync(d_next, 0, 16, s));
        WindowArgs g{a.ptr, a.idx, a.val, b.idx, b.val, seg, nw, t0, order + t0, nheavy, run,
                     off, hroff[c], tcol, tval, count, d_next};
        if (run > 0) {
            const int64_t ctas = std::min<int64_t>(std::max<int64_t>((run + Sh::kWarps - 1) / Sh::kWarps, g.nheavy),
                                                   (int64_t)num_sms() * Sh::kCtas);
            k_win_numeric<SR, T><<<(unsigned)ctas, 32 * Sh::kWarps, Sh::kSmem, s>>>(g);
            GBK_LAUNCHED();
        }
        GBK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, count, fin, nt + 1, s));
        count_launch(1);
        GBK_CUDA(cudaMemcpyAsync(&bcnt[c], fin + nt, 8, cudaMemcpyDeviceToHost, s));
        GBK_CUDA(cudaStreamSynchronize(s));
        GBK_REQUIRE(total + bcnt[c] < INT32_MAX, GBK_INVALID_VALUE, "gbk_mxm: the product has %lld entries or more (int32 limit)",
                    (long long)(total + bcnt[c]));
        const size_t entries = (size_t)std::max<int64_t>(bcnt[c], 1);
        if (nblocks == 1) {
            if (const int rc = own.get_entries(entries, sizeof(T))) return rc;
            bcol[c] = (int32_t*)own.p[1];
            bval[c] = (T*)own.p[2];
        } else if (dev.get(&bcol[c], 4 * entries) || dev.get(&bval[c], sizeof(T) * entries)) {
            set_error("gbk_mxm: out of device memory for a block's result");
            return GBK_OUT_OF_MEMORY;
        }
        if (bcnt[c] > 0) {
            k_win_gather<<<(unsigned)((nt + 7) / 8), 256, 0, s>>>(t0, nt, off, hroff[c], fin, tcol, (const uint32_t*)tval,
                                                                  bcol[c], (uint32_t*)bval[c]);
            GBK_LAUNCHED();
        }
        k_win_ptr<<<nb(cuts[c + 1] - cuts[c] + 1), 256, 0, s>>>(fin, cuts[c], cuts[c + 1] - cuts[c], nw, total,
                                                                (int32_t*)own.p[0]);
        GBK_LAUNCHED();
        total += bcnt[c];
    }
    if (nblocks > 1) {
        const size_t entries = (size_t)std::max<int64_t>(total, 1);
        if (const int rc = own.get_entries(entries, sizeof(T))) return rc;
        int64_t at = 0;
        for (size_t c = 0; c < nblocks; ++c) {
            if (bcnt[c] > 0) {
                GBK_CUDA(cudaMemcpyAsync((int32_t*)own.p[1] + at, bcol[c], 4 * (size_t)bcnt[c], cudaMemcpyDeviceToDevice, s));
                GBK_CUDA(cudaMemcpyAsync((T*)own.p[2] + at, bval[c], sizeof(T) * (size_t)bcnt[c], cudaMemcpyDeviceToDevice, s));
            }
            at += bcnt[c];
        }
    }
    const int rc = adopt_csr(out, n, m, total, (int32_t*)own.p[0], (int32_t*)own.p[1], own.p[2],
                             std::is_same<T, float>::value ? GBK_F32 : GBK_I32, s);
    if (rc) return rc;
    own.p[0] = own.p[1] = own.p[2] = nullptr;
    *done = true;
    return GBK_SUCCESS;
}

template <typename T>
int window_dispatch(gbk_matrix* out, const CsrView& a, const CsrView& b, int sr, int64_t block_entries, bool* done,
                    cudaStream_t s) {
    switch (sr) {
        case GBK_PLUS_TIMES: return window_t<GBK_PLUS_TIMES, T>(out, a, b, block_entries, done, s);
        case GBK_PLUS_SECOND: return window_t<GBK_PLUS_SECOND, T>(out, a, b, block_entries, done, s);
        case GBK_PLUS_ONE: return window_t<GBK_PLUS_ONE, T>(out, a, b, block_entries, done, s);
        case GBK_MIN_PLUS: return window_t<GBK_MIN_PLUS, T>(out, a, b, block_entries, done, s);
        case GBK_MIN_SECOND: return window_t<GBK_MIN_SECOND, T>(out, a, b, block_entries, done, s);
        case GBK_LOR_LAND: return window_t<GBK_LOR_LAND, T>(out, a, b, block_entries, done, s);
    }
    return GBK_SUCCESS;
}

}  // namespace

int mxm_window(gbk_matrix* out, const CsrView& a, const CsrView& b, int vtype, int sr, int64_t block_entries, bool* done,
               cudaStream_t s) {
    *done = false;
    if (a.nnz == 0 || b.nnz == 0 || b.ncols > kMaxColumns) return GBK_SUCCESS;
    return vtype == GBK_F32 ? window_dispatch<float>(out, a, b, sr, block_entries, done, s)
                            : window_dispatch<int32_t>(out, a, b, sr, block_entries, done, s);
}

}  // namespace gbk
