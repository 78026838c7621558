// kernels.cu -- bounds, binning, scans, compaction, conversions and
// transpose kernels of the Sp3MM library (sm_100a).  The per-row
// accumulation kernels are in rows.cu.
//
//  * Row binning by upper-bound size replaces the reference's OpenMP 1D / 2D
//    row and column partitions (code/src/Sp3MM_CSR_OMP_UB_Generic.c:85-105,
//    :153-182, :216-302): a bounds kernel gives each output row the number of
//    distinct keys its first table can receive (the reference's upper bound,
//    code/src/include/SpMMUtilsGeneric.h:112-139), and rows are grouped into
//    table-size levels by a count / scatter pair of kernels.
//  * The upper-bound flavour's merge (code/src/include/SpMMUtilsGeneric.h:
//    364-403) becomes a scan of the booked row lengths and a compaction kernel.
#include <cub/device/device_scan.cuh>

#include <atomic>
#include <climits>
#include <exception>
#include <type_traits>

#include "kernels.cuh"
#include "smem_limit.h"
#include "sp3mm_internal.cuh"

namespace sp3mm {

static std::atomic<uint64_t> g_launches{0};
uint64_t launch_count() { return g_launches.load(); }
void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

namespace {
struct SetSmemLimit {
    int operator()(const void* f, size_t bytes) const {
        return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(bytes));
    }
};
}  // namespace

cudaError_t raise_smem_limit(const void* f, size_t bytes) {
    // Never destroyed: a thread may launch while the process exits.
    static SmemLimits<SetSmemLimit>* limits = new SmemLimits<SetSmemLimit>(SetSmemLimit{});
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    try {
        return static_cast<cudaError_t>(limits->need(device, f, bytes));
    } catch (const std::exception&) {   // out of host memory
        return cudaErrorMemoryAllocation;
    }
}

__device__ __forceinline__ double load_val(const void* p, int vt, long long i) {
    if (vt == SP3MM_F32) return static_cast<double>(__ldg(static_cast<const float*>(p) + i));
    return __ldg(static_cast<const double*>(p) + i);
}
__device__ __forceinline__ void store_val(void* p, int vt, long long i, double v) {
    if (vt == SP3MM_F32) static_cast<float*>(p)[i] = __double2float_rn(v);
    else static_cast<double*>(p)[i] = v;
}

// ---------------------------------------------------------------------------
// Bounds.

// need[i] = min(flops_i, B.N) with flops_i = sum_{k in A(i)} len(B(k)).
template <int G>
__global__ void __launch_bounds__(256) k_pair_bounds(CsrView A, CsrView B, int* need,
                                                      unsigned long long* total) {
    const Group<G> g;
    const int groups = (gridDim.x * blockDim.x) / G;
    unsigned long long mine = 0;
    for (int row = (blockIdx.x * blockDim.x + threadIdx.x) / G; row < A.M; row += groups) {
        const int ab = __ldg(A.rp + row), ae = __ldg(A.rp + row + 1);
        long long f = 0;
        for (int t = ab + g.gl; t < ae; t += G) {
            const int k = __ldg(A.ci + t);
            f += __ldg(B.rp + k + 1) - __ldg(B.rp + k);
        }
        f = g.sum64(f);
        if (g.gl == 0) {
            const long long d = f < B.N ? f : B.N;
            need[row] = static_cast<int>(d < INT_MAX ? d : INT_MAX);
            mine += static_cast<unsigned long long>(f);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(total, mine);
}

// Direct R*A*P: need[i] = min(u1_i, A.N) with u1_i = sum_{k in R(i)} len(A(k))
// (the R*A row's products); total += u1_i * p_max_row, a bound on the C row's
// multiply-adds (each R*A entry forwards one P row of at most p_max_row
// entries).
template <int G>
__global__ void __launch_bounds__(256) k_direct_bounds(CsrView R, CsrView A, int p_max_row,
                                                        int* need, int* need_opt, int d1,
                                                        unsigned long long* total) {
    const Group<G> g;
    const int groups = (gridDim.x * blockDim.x) / G;
    unsigned long long mine = 0;
    for (int row = (blockIdx.x * blockDim.x + threadIdx.x) / G; row < R.M; row += groups) {
        const int rb = __ldg(R.rp + row), re = __ldg(R.rp + row + 1);
        long long u1 = 0;
        for (int t = rb + g.gl; t < re; t += G) {
            const int k = __ldg(R.ci + t);
            u1 += __ldg(A.rp + k + 1) - __ldg(A.rp + k);
        }
        u1 = g.sum64(u1);
        if (g.gl == 0) {
            const long long d = u1 < A.N ? u1 : A.N;
            need[row] = static_cast<int>(d < INT_MAX ? d : INT_MAX);
            if (need_opt) {
                // Optimistic first-table size: the bound >> d1, at most
                // 8 sqrt(products) -- long R*A rows repeat their columns
                // (stencil coarse levels: ~6 sqrt, kNN rows: <= 8.4 sqrt);
                // a row that overflows is recomputed with the bound.  A row
                // with at least as many products as A has columns is taken
                // as dense (the coarsest levels: every column, hundreds of
                // thousands of products) and gets the bound itself, which
                // bins it to the CTA-per-row kernel instead of a warp that
                // overflows and retries alone.
                long long o = d >> d1;
                const long long r =
                    static_cast<long long>(ceil(8.0 * sqrt(static_cast<double>(u1))));
                if (r < o) o = r;
                if (u1 >= A.N) o = d;
                if (d > 0 && o < 1) o = 1;
                need_opt[row] = static_cast<int>(o < INT_MAX ? o : INT_MAX);
            }
            mine += static_cast<unsigned long long>(u1) * static_cast<unsigned long long>(p_max_row);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(total, mine);
}

__global__ void k_need_from_counts(int M, const int* cnt, const int* cnt1, int* need) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M) return;
    int n = cnt[i];
    if (cnt1 && n > 0) n = max(n, cnt1[i]);
    need[i] = n;
}

// ---------------------------------------------------------------------------
// Binning by table-size level.

__host__ __device__ __forceinline__ int limit_of(long long S, int G) {
    const long long a = S - G - 1, b = (7 * S) / 8;
    return static_cast<int>(a < b ? a : b);
}

__host__ __device__ __forceinline__ int level_of(long long need, int G) {
    if (need <= 0) return -1;
    int L = 0;
    while (L < kLevels - 1 && limit_of(32ll << L, G) < need) ++L;
    return L;
}

int slots_for_need(long long need, int G) {
    const int L = level_of(need < 1 ? 1 : need, G);
    return 32 << L;
}
int level_for_need(long long need, int G) { return level_of(need, G); }

__global__ void __launch_bounds__(256) k_bin_levels(int M, const int* need, const int* est,
                                                     int shift, int G, signed char* level,
                                                     int* counts, int* nmax, int* row_cnt_zero) {
    __shared__ int sc[kLevels + 1];
    __shared__ int smax;
    for (int i = threadIdx.x; i <= kLevels; i += blockDim.x) sc[i] = 0;
    if (threadIdx.x == 0) smax = 0;
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
        const int n = need[i];
        int L = -1;
        if (n > 0) {
            const int s = est ? est[i] : n >> shift;
            L = level_of(s > 0 ? s : 1, G);
        }
        level[i] = static_cast<signed char>(L);
        if (L < 0) {
            atomicAdd(&sc[kLevels], 1);
            if (row_cnt_zero) row_cnt_zero[i] = 0;
        } else {
            atomicAdd(&sc[L], 1);
            atomicMax(&smax, n);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i <= kLevels; i += blockDim.x)
        if (sc[i]) atomicAdd(counts + i, sc[i]);
    if (threadIdx.x == 0 && smax) atomicMax(nmax, smax);
}

// Append every row to its level's list (cursors hold each list's start).
__global__ void __launch_bounds__(256) k_bin_scatter(int M, const signed char* level,
                                                      int* cursors, int* lists) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = i < M;
    const int L = in ? level[i] : -1;
    // Warp-aggregated append keeps the rows of a warp contiguous and ascending.
    const unsigned act = __ballot_sync(0xffffffffu, in && L >= 0);
    if (!(in && L >= 0)) return;
    const unsigned peers = __match_any_sync(act, L);
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(peers) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(cursors + L, __popc(peers));
    base = __shfl_sync(peers, base, leader);
    lists[base + __popc(peers & ((1u << lane) - 1u))] = i;
}

// ---------------------------------------------------------------------------
// Upper-bound flavour: copy of booked rows into exact CSR.  8 lanes per row.
__global__ void __launch_bounds__(256) k_compact(int M, const int* row_cnt,
                                                  const long long* row_off, const int* ub_ci,
                                                  const void* ub_v, const int* c_rp, int* c_ci,
                                                  void* c_v, int vt) {
    const Group<8> g;
    const int groups = (gridDim.x * blockDim.x) / 8;
    for (int row = (blockIdx.x * blockDim.x + threadIdx.x) / 8; row < M; row += groups) {
        const int n = row_cnt[row];
        if (!n) continue;
        const long long src = row_off[row];
        const long long dst = c_rp[row];
        for (int i = g.gl; i < n; i += 8) {
            c_ci[dst + i] = ub_ci[src + i];
            if (vt == SP3MM_F32)
                static_cast<float*>(c_v)[dst + i] = static_cast<const float*>(ub_v)[src + i];
            else
                static_cast<double*>(c_v)[dst + i] = static_cast<const double*>(ub_v)[src + i];
        }
    }
}

// ---------------------------------------------------------------------------
// Conversions between the host ABI (64-bit, OFF_F based) and device CSR.

__global__ void k_narrow_rowptr(long long M, long long nnz, const unsigned long long* src,
                                int off, int* dst, unsigned* err) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i <= M;
         i += (long long)gridDim.x * blockDim.x) {
        const long long v = static_cast<long long>(src[i]) - off;
        bool bad = v < 0 || v > nnz;
        if (i == 0) bad |= v != 0;
        if (i == M) bad |= v != nnz;
        if (i > 0) bad |= static_cast<long long>(src[i - 1]) - off > v;
        if (bad) atomicOr(err, kErrInput);
        dst[i] = static_cast<int>(bad ? 0 : v);
    }
}

// Warp per row: narrow columns, check range and strict ascending order.
__global__ void __launch_bounds__(256) k_narrow_cols(long long M, long long N, const int* rp,
                                                      const unsigned long long* src, int off,
                                                      int* dst, int* max_row, unsigned* err) {
    const int lane = threadIdx.x & 31;
    const long long warps = (gridDim.x * (long long)blockDim.x) / 32;
    int my_max = 0;
    for (long long row = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / 32; row < M;
         row += warps) {
        const int b = rp[row], e = rp[row + 1];
        my_max = max(my_max, e - b);
        for (int j = b + lane; j < e; j += 32) {
            const long long c = static_cast<long long>(src[j]) - off;
            bool bad = c < 0 || c >= N;
            if (j > b) bad |= static_cast<long long>(src[j - 1]) - off >= c;
            if (bad) atomicOr(err, kErrInput);
            dst[j] = static_cast<int>(bad ? 0 : c);
        }
    }
    if (lane == 0 && my_max) atomicMax(max_row, my_max);
}

__global__ void k_widen(long long n, const int* src, int off, unsigned long long* dst) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        dst[i] = static_cast<unsigned long long>(static_cast<long long>(src[i]) + off);
}

__global__ void k_convert_values(long long n, const void* src, int st_, void* dst, int dt) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        store_val(dst, dt, i, load_val(src, st_, i));
}

// Validate a device-side int32 CSR: row_ptr monotone from 0, columns in
// range and strictly ascending within rows.
__global__ void __launch_bounds__(256) k_validate_i32(int M, int N, const int* rp,
                                                       const int* ci, int* max_row,
                                                       unsigned* err) {
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) / 32;
    int my_max = 0;
    for (int row = (blockIdx.x * blockDim.x + threadIdx.x) / 32; row < M; row += warps) {
        const int b = rp[row], e = rp[row + 1];
        if (e < b || (row == 0 && b != 0)) {
            if (lane == 0) atomicOr(err, kErrInput);
            continue;
        }
        my_max = max(my_max, e - b);
        for (int j = b + lane; j < e; j += 32) {
            const int c = ci[j];
            bool bad = c < 0 || c >= N;
            if (j > b) bad |= ci[j - 1] >= c;
            if (bad) atomicOr(err, kErrInput);
        }
    }
    if (lane == 0 && my_max) atomicMax(max_row, my_max);
}

// ---------------------------------------------------------------------------
// Transpose.

__global__ void k_col_counts(long long nnz, const int* ci, int* counts) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nnz;
         i += (long long)gridDim.x * blockDim.x)
        atomicAdd(counts + ci[i], 1);
}

// 2^lg lanes per row of A (its mean length: a warp per row of the four
// entries of a fine prolongator took 0.41 ms at 128^3, four lanes 0.09), and
// the whole warp for a row of more than kScatterLong times its lanes (a row of
// 200,000 entries among 500,000 of two: 19.6 ms on two lanes, 3.4 on a warp).
constexpr int kScatterLong = 8;
__global__ void __launch_bounds__(256) k_transpose_scatter(CsrView A, int lg, const int* t_rp,
                                                             int* cursor, int* t_ci, void* t_v) {
    const int lane = threadIdx.x & 31;
    const int sub = lane & ((1 << lg) - 1);
    auto scatter = [&](int row, int b, int e, int step) {
        for (int j = b; j < e; j += step) {
            const int c = A.ci[j];
            const int pos = t_rp[c] + atomicAdd(cursor + c, 1);
            t_ci[pos] = row;
            if (A.vtype == SP3MM_F32)
                static_cast<float*>(t_v)[pos] = static_cast<const float*>(A.v)[j];
            else
                static_cast<double*>(t_v)[pos] = static_cast<const double*>(A.v)[j];
        }
    };
    const long long groups = (static_cast<long long>(gridDim.x) * blockDim.x) >> lg;
    // (row - (lane >> lg): the warp's first row, the same for all its lanes)
    for (long long row = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> lg;
         row - (lane >> lg) < A.M; row += groups) {
        int b = 0, e = 0;
        if (row < A.M) {
            b = A.rp[row];
            e = A.rp[row + 1];
        }
        const bool big = e - b > kScatterLong << lg;
        if (!big) scatter(static_cast<int>(row), b + sub, e, 1 << lg);
        for (unsigned m = __ballot_sync(0xffffffffu, big && sub == 0); m; m &= m - 1) {
            const int src = __ffs(m) - 1;
            const int r = __shfl_sync(0xffffffffu, static_cast<int>(row), src);
            const int rb = __shfl_sync(0xffffffffu, b, src);
            const int re = __shfl_sync(0xffffffffu, e, src);
            scatter(r, rb + lane, re, 32);
        }
    }
}

// Rows of more than 32 and at most kSortSmemRow entries: a CTA per row counts
// every column's rank (the row in shared memory, four columns compared per
// load).  The coarse levels' restrictions hold rows of 84 to 677 entries: a
// warp per row with a bitonic network took 1.13 ms over the levels of a 128^3
// hierarchy, this 0.43.  Ranks take n^2 comparisons: rows past kSortRankRow
// entries go to a launch of their own (NET), a bitonic network of one size by
// the CTA (transpose with 1,000 rows of 2,000: 1.28 -> 0.46 ms; both in one
// kernel made rows of 700 8 % slower).  A column met twice is flagged where err
// is given.
constexpr int kSortSmemRow = 2048;
static_assert(kSortRankRow == kSortSmemRow / 2, "the network's one size");
constexpr int kSortThreads = 128;

// Bitonic network over kSortSmemRow keys.
__device__ __forceinline__ void sort_network(unsigned long long* key) {
    for (int k = 2; k <= kSortSmemRow; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            __syncthreads();
            for (int q = threadIdx.x; q < kSortSmemRow / 2; q += kSortThreads) {
                const int i = 2 * q - (q & (j - 1));
                const unsigned long long a = key[i], c = key[i + j];
                if ((a > c) == ((i & k) == 0)) {
                    key[i] = c;
                    key[i + j] = a;
                }
            }
        }
    }
    __syncthreads();
}

// A row of n > kSortRankRow entries from b on: its columns are sorted with
// their places, then the values fetched from there into the keys' storage
// (before any is overwritten) and written.
__device__ __forceinline__ void sort_row_network(unsigned long long* key, int b, int n, int* ci,
                                                 void* v, int vt, unsigned* err) {
    static_assert(kSortSmemRow == 2048, "places take 11 bits");
    for (int i = threadIdx.x; i < kSortSmemRow; i += kSortThreads)
        key[i] = i < n ? static_cast<unsigned long long>(ci[b + i]) << 11 | i : ~0ULL;
    sort_network(key);
    for (int i = threadIdx.x; i < n; i += kSortThreads) {
        ci[b + i] = static_cast<int>(key[i] >> 11);
        if (i > 0 && key[i - 1] >> 11 == key[i] >> 11 && err) atomicOr(err, kErrInput);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += kSortThreads)
        key[i] = __double_as_longlong(load_val(v, vt, b + static_cast<int>(key[i] & 2047)));
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += kSortThreads)
        store_val(v, vt, b + i, __longlong_as_double(key[i]));
    __syncthreads();
}

// A row of n > 32 entries from b on by ranks.
__device__ __forceinline__ void sort_row_ranks(int* sk, double* sv, int b, int n, int* ci,
                                               void* v, int vt, unsigned* err) {
    constexpr int U = 4;   // columns a thread ranks together
    for (int i = threadIdx.x; i < n; i += kSortThreads) {
        sk[i] = ci[b + i];
        sv[i] = load_val(v, vt, b + i);
    }
    if (threadIdx.x < 4) sk[n + threadIdx.x] = INT_MAX;
    __syncthreads();
    for (int i0 = threadIdx.x; i0 < n; i0 += U * kSortThreads) {
        int k[U], lt[U], eq[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u * kSortThreads;
            k[u] = i < n ? sk[i] : -1;
            lt[u] = eq[u] = 0;
        }
        for (int j = 0; j < n; j += 4) {
            const int4 q = *reinterpret_cast<const int4*>(sk + j);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (u * kSortThreads < n) {
                    lt[u] += (q.x < k[u]) + (q.y < k[u]) + (q.z < k[u]) + (q.w < k[u]);
                    eq[u] += (q.x == k[u]) + (q.y == k[u]) + (q.z == k[u]) + (q.w == k[u]);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u * kSortThreads;
            if (i < n) {
                ci[b + lt[u]] = k[u];
                store_val(v, vt, b + lt[u], sv[i]);
                if (eq[u] > 1 && err) atomicOr(err, kErrInput);
            }
        }
    }
    __syncthreads();
}

template <bool NET>
__global__ void __launch_bounds__(kSortThreads) k_sort_rows_cta(int M, int chunk, const int* rp,
                                                                int* ci, void* v, int vt,
                                                                unsigned* err) {
    constexpr int kMin = NET ? kSortRankRow : 32, kMax = NET ? kSortSmemRow : kSortRankRow;
    __shared__ __align__(16) int sk[NET ? 4 : kMax + 4];
    __shared__ std::conditional_t<NET, unsigned long long, double> sv[kMax];
    const int lane = threadIdx.x & 31;
    for (long long r0 = blockIdx.x * static_cast<long long>(chunk); r0 < M;
         r0 += gridDim.x * static_cast<long long>(chunk)) {
        // Every warp looks the chunk's (at most 32) lengths up.
        int lb = 0, ln = 0;
        if (lane < chunk && r0 + lane < M) {
            lb = rp[r0 + lane];
            ln = rp[r0 + lane + 1] - lb;
        }
        unsigned rows = __ballot_sync(0xffffffffu, ln > kMin && ln <= kMax);
        for (; rows; rows &= rows - 1) {
            const int b = __shfl_sync(0xffffffffu, lb, __ffs(rows) - 1);
            const int n = __shfl_sync(0xffffffffu, ln, __ffs(rows) - 1);
            if constexpr (NET) sort_row_network(sv, b, n, ci, v, vt, err);
            else sort_row_ranks(sk, sv, b, n, ci, v, vt, err);
        }
    }
}

// Sort each row's (col, val) by col.  Warp per row; rows up to 32 entries by
// rank in registers, rows of k_sort_rows_cta's range there, longer rows by
// odd-even transposition in place.
__global__ void __launch_bounds__(256) k_sort_rows(int M, const int* rp, int* ci, void* v,
                                                    int vt, unsigned* err) {
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) / 32;
    for (int row = (blockIdx.x * blockDim.x + threadIdx.x) / 32; row < M; row += warps) {
        const int b = rp[row], e = rp[row + 1];
        const int n = e - b;
        if (n <= 1) continue;
        if (n <= 32) {
            const bool in = lane < n;
            const int k = in ? ci[b + lane] : INT_MAX;
            const double x = in ? load_val(v, vt, b + lane) : 0.0;
            int r = 0, eq = 0;
            for (int j = 0; j < n; ++j) {
                const int kj = __shfl_sync(0xffffffffu, k, j);
                r += kj < k;
                eq += kj == k;
            }
            __syncwarp();
            if (in) {
                ci[b + r] = k;
                store_val(v, vt, b + r, x);
                if (eq > 1 && err) atomicOr(err, kErrInput);
            }
            __syncwarp();
            continue;
        }
        if (n <= kSortSmemRow) continue;   // k_sort_rows_cta
        for (int phase = 0; phase < n; ++phase) {
            for (int i = b + (phase & 1) + 2 * lane; i + 1 < e; i += 64) {
                const int a0 = ci[i], a1 = ci[i + 1];
                if (a0 > a1) {
                    ci[i] = a1;
                    ci[i + 1] = a0;
                    const double x0 = load_val(v, vt, i), x1 = load_val(v, vt, i + 1);
                    store_val(v, vt, i, x1);
                    store_val(v, vt, i + 1, x0);
                }
            }
            __syncwarp();
        }
        if (err)
            for (int i = b + lane; i + 1 < e; i += 32)
                if (ci[i] == ci[i + 1]) atomicOr(err, kErrInput);
    }
}

// ---------------------------------------------------------------------------
// 2D column-partition upper bounds (code/src/include/SpMMUtilsGeneric.h:146-174).
__global__ void k_colparts_ub(CsrView A, int gridCols, const long long* off, long long* out,
                              unsigned long long* total) {
    unsigned long long mine = 0;
    for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x;
         x < static_cast<long long>(A.M) * gridCols; x += (long long)gridDim.x * blockDim.x) {
        const int r = static_cast<int>(x / gridCols);
        const int gc = static_cast<int>(x % gridCols);
        long long s = 0;
        for (int jj = A.rp[r]; jj < A.rp[r + 1]; ++jj) {
            const long long id = static_cast<long long>(A.ci[jj]) * gridCols + gc;
            s += off[id + 1] - off[id];
        }
        out[x] = s;
        mine += static_cast<unsigned long long>(s);
    }
    if (mine) atomicAdd(total, mine);
}

// ---------------------------------------------------------------------------
// Host launchers.

static inline int grid_for(long long work, int block, int cap = 148 * 16) {
    long long g = (work + block - 1) / block;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return static_cast<int>(g);
}

void launch_pair_bounds(const CsrView& A, const CsrView& B, int* need,
                        unsigned long long* total, cudaStream_t st) {
    if (A.M == 0) return;
    k_pair_bounds<8><<<grid_for(static_cast<long long>(A.M) * 8, 256), 256, 0, st>>>(A, B, need,
                                                                                     total);
    note_launch();
}

void launch_direct_bounds(const CsrView& R, const CsrView& A, int p_max_row, int* need,
                          unsigned long long* total, cudaStream_t st, int* need_opt, int d1) {
    if (R.M == 0) return;
    k_direct_bounds<8><<<grid_for(static_cast<long long>(R.M) * 8, 256), 256, 0, st>>>(
        R, A, p_max_row, need, need_opt, d1, total);
    note_launch();
}

__global__ void k_count_max(int M, const int* cnt, const int* rp, int* out,
                            unsigned long long* sum) {
    int m = 0;
    unsigned long long t = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
        const int c = cnt ? cnt[i] : rp[i + 1] - rp[i];
        m = max(m, c);
        t += static_cast<unsigned long long>(c);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (m > 0) atomicMax(out, m);
        if (sum && t) atomicAdd(sum, t);
    }
}

void launch_count_max(int M, const int* cnt, const int* rp, int* out, cudaStream_t st,
                      unsigned long long* sum) {
    if (M == 0) return;
    k_count_max<<<grid_for(M, 256), 256, 0, st>>>(M, cnt, rp, out, sum);
    note_launch();
}

void launch_need_from_counts(int M, const int* cnt, const int* cnt1, int* need,
                             cudaStream_t st) {
    if (M == 0) return;
    k_need_from_counts<<<(M + 255) / 256, 256, 0, st>>>(M, cnt, cnt1, need);
    note_launch();
}

void launch_bin_levels(int M, const int* need, int shift, int G, signed char* level,
                       int* counts, int* nmax, int* row_cnt_zero, cudaStream_t st,
                       const int* est) {
    if (M == 0) return;
    k_bin_levels<<<grid_for(M, 256), 256, 0, st>>>(M, need, est, shift, G, level, counts, nmax,
                                                    row_cnt_zero);
    note_launch();
}

void launch_bin_scatter(int M, const signed char* level, int* cursors, int* lists,
                        cudaStream_t st) {
    if (M == 0) return;
    k_bin_scatter<<<(M + 255) / 256, 256, 0, st>>>(M, level, cursors, lists);
    note_launch();
}

void launch_compact(int M, const int* row_cnt, const long long* row_off, const int* ub_ci,
                    const void* ub_v, const int* c_rp, int* c_ci, void* c_v, int vt,
                    cudaStream_t st) {
    if (M == 0) return;
    k_compact<<<grid_for(static_cast<long long>(M) * 8, 256), 256, 0, st>>>(
        M, row_cnt, row_off, ub_ci, ub_v, c_rp, c_ci, c_v, vt);
    note_launch();
}

size_t scan_temp_bytes(int M) {
    size_t bytes = 0;
    cub::DeviceScan::InclusiveSum(nullptr, bytes, static_cast<const int*>(nullptr),
                                  static_cast<int*>(nullptr), M > 0 ? M : 1);
    return bytes;
}

void launch_scan(int M, const int* cnt, int* row_ptr, void* temp, size_t temp_bytes,
                 cudaStream_t st) {
    cudaMemsetAsync(row_ptr, 0, sizeof(int), st);
    if (M == 0) return;
    cub::DeviceScan::InclusiveSum(temp, temp_bytes, cnt, row_ptr + 1, M, st);
    note_launch();
}

void launch_narrow_rowptr(long long M, long long nnz, const unsigned long long* src, int off,
                          int* dst, unsigned* err, cudaStream_t st) {
    k_narrow_rowptr<<<grid_for(M + 1, 256), 256, 0, st>>>(M, nnz, src, off, dst, err);
    note_launch();
}

void launch_narrow_cols(long long M, long long N, const int* rp, const unsigned long long* src,
                        int off, int* dst, int* max_row, unsigned* err, cudaStream_t st) {
    if (M == 0) return;
    k_narrow_cols<<<grid_for(M * 32, 256), 256, 0, st>>>(M, N, rp, src, off, dst, max_row,
                                                         err);
    note_launch();
}

void launch_widen(long long n, const int* src, int off, unsigned long long* dst,
                  cudaStream_t st) {
    if (n == 0) return;
    k_widen<<<grid_for(n, 256), 256, 0, st>>>(n, src, off, dst);
    note_launch();
}

void launch_convert_values(long long n, const void* src, int src_type, void* dst, int dst_type,
                           cudaStream_t st) {
    if (n == 0) return;
    k_convert_values<<<grid_for(n, 256), 256, 0, st>>>(n, src, src_type, dst, dst_type);
    note_launch();
}

void launch_validate_i32(int M, int N, const int* rp, const int* ci, int* max_row,
                         unsigned* err, cudaStream_t st) {
    if (M == 0) return;
    k_validate_i32<<<grid_for(static_cast<long long>(M) * 32, 256), 256, 0, st>>>(
        M, N, rp, ci, max_row, err);
    note_launch();
}

void launch_col_counts(long long nnz, const int* ci, int* counts, cudaStream_t st) {
    if (nnz == 0) return;
    k_col_counts<<<grid_for(nnz, 256), 256, 0, st>>>(nnz, ci, counts);
    note_launch();
}

void launch_transpose_scatter(const CsrView& A, const int* t_rp, int* cursor, int* t_ci,
                              void* t_v, cudaStream_t st) {
    if (A.M == 0) return;
    int lg = 0;
    while (lg < 5 && (1LL << lg) * A.M < A.nnz) ++lg;   // mean row length
    k_transpose_scatter<<<grid_for(static_cast<long long>(A.M) << lg, 256), 256, 0, st>>>(
        A, lg, t_rp, cursor, t_ci, t_v);
    note_launch();
}

namespace {
// CTAs of a row sort and the row lengths each looks up at once: few rows one by
// one, many 32 at a time.
struct SortGrid {
    int grid, chunk;
};
SortGrid sort_grid(int M) {
    const int ctas = 148 * 8;
    const int chunk = M < ctas ? 1 : M / ctas < 32 ? M / ctas : 32;
    return {grid_for(M, chunk, ctas), chunk};
}
}  // namespace

void launch_sort_rows(int M, const int* rp, int* ci, void* v, int vt, int max_row,
                      cudaStream_t st, unsigned* err) {
    if (M == 0 || max_row <= 1) return;
    k_sort_rows<<<grid_for(static_cast<long long>(M) * 32, 256), 256, 0, st>>>(M, rp, ci, v, vt,
                                                                              err);
    note_launch();
    if (max_row > 32) {
        const SortGrid g = sort_grid(M);
        k_sort_rows_cta<false><<<g.grid, kSortThreads, 0, st>>>(M, g.chunk, rp, ci, v, vt, err);
        note_launch();
    }
    if (max_row > kSortRankRow) launch_sort_long_rows(M, rp, ci, v, vt, st, err);
}

void launch_sort_long_rows(int M, const int* rp, int* ci, void* v, int vt, cudaStream_t st,
                           unsigned* err) {
    const SortGrid g = sort_grid(M);
    k_sort_rows_cta<true><<<g.grid, kSortThreads, 0, st>>>(M, g.chunk, rp, ci, v, vt, err);
    note_launch();
}

void launch_colparts_ub(const CsrView& A, int gridCols, const long long* bColOffsets,
                        long long* out, unsigned long long* total, cudaStream_t st) {
    const long long work = static_cast<long long>(A.M) * gridCols;
    if (work == 0) return;
    k_colparts_ub<<<grid_for(work, 256), 256, 0, st>>>(A, gridCols, bColOffsets, out, total);
    note_launch();
}

}  // namespace sp3mm
