// rowtiny.cuh -- SpMM rows of at most kTinyProducts products, one thread per
// row (sm_100a).
//
// A warp per row leaves most lanes idle when a row has 7 to 32 products (A*P
// on a fine stencil level: 15 or 28), and a few lanes per row pay the probes
// and ballots of a hash table for them.  Here each thread walks its row's
// products in the reference's order -- left position t ascending, then the
// selected right row's entries ascending
// (code/src/include/SpMMUtilsGeneric.h:39-55) -- and keeps the distinct
// columns as a list in shared memory, searched linearly (the lists of a CTA's
// threads are interleaved, so a step of the search is one conflict-free
// access for the warp).  A warp's rows are then sorted by counting and
// written together, in consecutive places.
//
// A*P, 96x80x88 7-point box (675,840 rows of 28 products): 0.25 ms against
// 0.60 on a warp per row and 0.39 on four lanes per row; 900x800 5-point grid
// (720,000 rows of 15): 0.10 against 0.56 and 0.31; A*P0 at 128^3 (7 products):
// 0.15 against 0.85 on four lanes.  Bound by the searches' shared-memory
// latency; past 32 products the quadratic search would lose to a table.
#pragma once

#include "rowwarp.cuh"

namespace sp3mm {

constexpr int kTinyThreads = 128;

// Shared memory of a CTA: vals keys ranks, `cap` entries per thread.
__host__ __device__ __forceinline__ size_t tiny_bytes(bool num, int cap) {
    return static_cast<size_t>(cap) * kTinyThreads * (num ? 13 : 4);
}

template <int MODE, typename TV, typename TO>
__global__ void __launch_bounds__(kTinyThreads) k_pair_tiny(PairRowArgs a, RowParams p) {
    constexpr bool NUM = MODE != kSymb;
    constexpr int T = kTinyThreads;
    extern __shared__ __align__(16) unsigned char smem[];
    const int cap = p.S1;
    double* vals = reinterpret_cast<double*>(smem) + threadIdx.x;
    int* keys = reinterpret_cast<int*>(smem + (NUM ? static_cast<size_t>(cap) * T * 8 : 0)) +
                threadIdx.x;
    unsigned char* at = reinterpret_cast<unsigned char*>(keys - threadIdx.x + cap * T);
    const int lane = threadIdx.x & 31;
    const TV* avals = static_cast<const TV*>(a.A.v);
    const TV* bvals = static_cast<const TV*>(a.B.v);
    for (long long r0 = static_cast<long long>(blockIdx.x) * T + (threadIdx.x & ~31);
         r0 < p.nrows; r0 += static_cast<long long>(gridDim.x) * T) {
        const int row = static_cast<int>(r0) + lane;
        const bool has = row < p.nrows;
        int n = 0;
        if (has) {
            const int e0 = __ldg(a.A.rp + row), e1 = __ldg(a.A.rp + row + 1);
            for (int t = e0; t < e1; ++t) {
                const int k = __ldg(a.A.ci + t);
                const double s = NUM ? ldv(avals, t) : 0.0;
                const int b1 = __ldg(a.B.rp + k + 1);
                for (int e = __ldg(a.B.rp + k); e < b1; ++e) {
                    const int c = __ldg(a.B.ci + e);
                    int m = n;
                    for (int i = 0; i < n; ++i)
                        if (keys[i * T] == c) m = i;
                    if (m == n) {
                        if (n == cap) {   // more products than the longest rows allow
                            atomicOr(p.err, kErrInput);
                            break;
                        }
                        keys[n * T] = c;
                        if (NUM) vals[n * T] = 0.0;
                        ++n;
                    }
                    if (NUM)
                        vals[m * T] =
                            __dadd_rn(vals[m * T], __dmul_rn(ldv(bvals, e), s));
                }
            }
        }
        if constexpr (!NUM) {
            if (has) p.row_cnt[row] = n;
        } else {
            // Entry i of this thread goes to place rank(i): at[rank * T] = i.
            for (int i = 0; i < n; ++i) {
                const int c = keys[i * T];
                int r = 0;
                for (int j = 0; j < n; ++j) r += keys[j * T] < c;
                at[r * T + threadIdx.x] = static_cast<unsigned char>(i);
            }
            int total;
            const int first = wscan_excl(n, total);
            long long base = -1;
            if (MODE == kNumBook) {
                unsigned long long b = 0;
                if (lane == 0 && total) b = atomicAdd(p.cursor, static_cast<unsigned long long>(total));
                b = __shfl_sync(kFull, b, 0);
                if (b + total > p.cap) {
                    if (lane == 0) atomicOr(p.err, kErrBook);
                } else {
                    base = static_cast<long long>(b) + first;
                    if (has) {
                        p.row_off[row] = base;
                        p.row_cnt[row] = n;
                    }
                }
            } else if (has) {
                base = p.c_rp[row];
                if (p.c_rp[row + 1] - base != n) {
                    atomicOr(p.err, kErrCount);
                    base = -1;
                }
            }
            __syncwarp();
            int* oc = MODE == kNumBook ? p.ub_ci : p.c_ci;
            TO* ov = static_cast<TO*>(MODE == kNumBook ? p.ub_v : p.c_v);
            for (int f0 = 0; f0 < total; f0 += 32) {
                const int f = f0 + lane;
                // The last thread whose first entry is at or before f.
                int j = 0;
#pragma unroll
                for (int step = 16; step > 0; step >>= 1) {
                    const int o = __shfl_sync(kFull, first, j + step);
                    if (o <= f) j += step;
                }
                const int i = f - __shfl_sync(kFull, first, j);
                const long long b = __shfl_sync(kFull, base, j);
                if (f < total && b >= 0) {
                    const int d = j - lane;   // that thread's lists
                    const int m = at[i * T + threadIdx.x + d] * T + d;
                    oc[b + i] = keys[m];
                    stv(ov, b + i, vals[m]);
                }
            }
            __syncwarp();
        }
    }
}

}  // namespace sp3mm
