// rowreplay.cuh -- rows of few products whose column patterns repeat, summed
// from one worked-out pattern (sm_100a).
//
// A row's sums are fixed by which of its products meet in a column.  A CTA
// takes a run of consecutive rows and works that out once, for a row of the
// most frequent length among 32 spread over its run (replay_pick): per stage,
// the template holds the products in the reference's order -- left position t
// ascending, then the selected right row's entries ascending
// (code/src/include/SpMMUtilsGeneric.h:39-55) -- with their columns and, per
// distinct column, the list of its products in that order.  Another row whose
// right rows have the same lengths and whose product columns are the
// template's plus one constant meets in the same places, whatever its values:
// that is checked, product by product, as the products are loaded.  On the
// inside of a structured grid nearly every row passes; the others go to a list
// that the register-product kernels run (rowlanes.cuh).
//
// The sums then need no table: each lane owns a column and adds its listed
// products one after another, from 0.0, in the reference's order, so values
// are bit-identical.  Stage 1 of the direct product lists its columns in
// first-touch order (code/src/include/sparseMatrix.h:85-104), the order in
// which it forwards them into P
// (code/src/Sp3MM_CSR_OMP_UB_Generic.c:542-545); the last stage lists them
// ascending, so the row is written straight from the sums.
//
// Why: the table kernels spend about 7 warp instructions a product on finding
// which products meet; this one spends 1.3 (79 M for 110,592 rows of a 96^3
// 7-point box, 558 products each).  128^3: 0.66 ms for the 218,000 rows that
// match (boundary rows up to two coarse cells deep do not), 0.29 ms on the
// lanes kernel for the rest, against 1.51 ms for all of them there; the
// symbolic pass 0.28 + 0.19 against 1.05 ms.  Bound by the latency of the
// loads' chain (left row, its bounds, the entries, twice) at 17 warps an SM
// and by the L1 data stage (62 %: half of it the sums' gathers), so two rows
// share every index read, four batches are loaded ahead, and the lanes of a
// round get columns with lists of about one length.  Measured and not kept:
// one row at a time (0.83-1.0 ms), four (0.78: too few warps fit), a template
// per warp (1.1: half the warps).
#pragma once

#include "batch.cuh"
#include "rowwarp.cuh"

namespace sp3mm {

// Slots of the build's hash table: at least twice the columns, and room for
// one more batch of 32 new ones past the capacity.
__host__ __device__ __forceinline__ int replay_hash(int ns) {
    int S = 64;
    while (S < 2 * ns || S < ns + 64) S <<= 1;
    return S;
}

// One stage's template (shared memory) and its sizes (registers, warp-uniform).
struct ReplayStage {
    int* tc;               // [npcap] product columns
    int* sc;               // [nscap] distinct columns
    unsigned short* gidx;  // [npcap] products by column
    unsigned short* gst;   // [nscap + 1] each column's first in gidx
    unsigned short* off;   // [kcap + 1] each step's first product
    unsigned char* perm;   // [nscap] columns by falling product count
    unsigned char* tk;     // [npcap] step of each product
    int npcap, nscap, kcap;
    int np, ns, nst;       // products, columns, steps (-1: no template)
};

// Rows that a warp replays together.  Their working arrays are interleaved,
// so that one 16-byte access serves both rows.
constexpr int kReplayRows = 2;

// A warp's working arrays, and the template build's scratch (a CTA's only; it
// lies over the working arrays).
struct ReplayScratch {
    double2* prod;          // [npm] rounded products
    double2* ss;            // [k1] stage 1's left values
    double2* rav;           // [ns1] stage 1's sums, stage 2's left values
    int2* sb;               // [km] right-row start minus product offset
    int* sb1;               // [km] the same of the template's row
    int* hk;                // [hash] keys
    unsigned char* hv;      // [hash] and columns' numbers
    int hmask, hshift;
    int* rk;                // columns in first-touch order
    unsigned short* rc;     // and their product counts
    unsigned char* rid;     // and their final numbers
    unsigned short* tmp;    // [npm] column number and place in it
};

struct ReplayLayout {
    size_t bytes = 0;
    __host__ __device__ __forceinline__ size_t take(size_t n, size_t align) {
        bytes = (bytes + align - 1) / align * align;
        const size_t at = bytes;
        bytes += n;
        return at;
    }
};
// Shared memory of a CTA of `warps` warps (base null: size only).
__host__ __device__ __forceinline__ size_t replay_place(const ReplayCaps& c, bool num, int warps,
                                                        int warp, unsigned char* base,
                                                        ReplayStage* st, ReplayScratch* sx) {
    const bool direct = c.np2 > 0;
    const int npm = c.np1 > c.np2 ? c.np1 : c.np2;
    const int nsm = c.ns1 > c.ns2 ? c.ns1 : c.ns2;
    const int km = direct && c.ns1 > c.k1 ? c.ns1 : c.k1;
    const int H = replay_hash(nsm);
    ReplayLayout l;
    size_t tc[2], gi[2], gs[2], of[2], tk[2], sc[2], pm[2];
    const int np[2] = {c.np1, c.np2}, ns[2] = {c.ns1, c.ns2}, k[2] = {c.k1, direct ? c.ns1 : 0};
    for (int i = 0; i < 2; ++i) tc[i] = l.take(4 * static_cast<size_t>(np[i]), 4);
    for (int i = 0; i < 2; ++i) sc[i] = l.take(4 * static_cast<size_t>(ns[i]), 4);
    for (int i = 0; i < 2; ++i) {
        gi[i] = l.take(2 * static_cast<size_t>(np[i]), 2);
        gs[i] = l.take(2 * static_cast<size_t>(ns[i] + 1), 2);
        of[i] = l.take(2 * static_cast<size_t>(k[i] + 1), 2);
    }
    for (int i = 0; i < 2; ++i) {
        tk[i] = l.take(static_cast<size_t>(np[i]), 1);
        pm[i] = l.take(static_cast<size_t>(ns[i]), 1);
    }
    // Working arrays of every warp.
    ReplayLayout w;
    const size_t prod = w.take(num ? 16 * static_cast<size_t>(npm) : 0, 16);
    const size_t rav = w.take(num && direct ? 16 * static_cast<size_t>(c.ns1) : 0, 16);
    const size_t ss = w.take(num ? 16 * static_cast<size_t>(c.k1) : 0, 16);
    const size_t sb = w.take(8 * static_cast<size_t>(km), 8);
    const size_t per_warp = (w.take(0, 16), w.bytes);
    // Build scratch.
    ReplayLayout b;
    const size_t sb0 = b.take(4 * static_cast<size_t>(km), 4);
    const size_t hk = b.take(4 * static_cast<size_t>(H), 4);
    const size_t hv = b.take(static_cast<size_t>(H), 1);
    const size_t rk = b.take(4 * static_cast<size_t>(nsm + 3), 16);
    const size_t rc = b.take(2 * static_cast<size_t>(nsm), 2);
    const size_t tmp = b.take(2 * static_cast<size_t>(npm), 2);
    const size_t rid = b.take(static_cast<size_t>(nsm), 1);
    const size_t work = l.take(0, 16);
    const size_t all = static_cast<size_t>(warps) * per_warp;
    const size_t total = (work + (all > b.bytes ? all : b.bytes) + 15) / 16 * 16;
    if (base) {
        auto u16 = [&](size_t o) { return reinterpret_cast<unsigned short*>(base + o); };
        auto i32 = [&](size_t o) { return reinterpret_cast<int*>(base + o); };
        if (st)
#pragma unroll
            for (int i = 0; i < 2; ++i)
                st[i] = ReplayStage{i32(tc[i]), i32(sc[i]), u16(gi[i]), u16(gs[i]), u16(of[i]),
                                base + pm[i], base + tk[i], np[i], ns[i], k[i], 0, 0, -1};
        const size_t own = work + static_cast<size_t>(warp) * per_warp;
        sx->prod = reinterpret_cast<double2*>(base + own + prod);
        sx->rav = reinterpret_cast<double2*>(base + own + rav);
        sx->ss = reinterpret_cast<double2*>(base + own + ss);
        sx->sb = reinterpret_cast<int2*>(base + own + sb);
        sx->sb1 = i32(work + sb0);
        sx->hk = i32(work + hk);
        sx->hv = base + work + hv;
        sx->hmask = H - 1;
        sx->hshift = 32 - ilog2_pow2(static_cast<unsigned>(H));
        sx->rk = i32(work + rk);
        sx->rc = u16(work + rc);
        sx->rid = base + work + rid;
        sx->tmp = u16(work + tmp);
    }
    return total;
}

// Left row's columns.
struct LeftR {
    const int* keys;
    __device__ __forceinline__ int key(int t) const { return keys[t]; }
};

// Column lists of the template's products tc[0..np): columns numbered in
// first-touch order, or ascending (SORTED).  False when they do not fit.
template <bool SORTED>
__device__ __forceinline__ bool replay_build(ReplayStage& st, const ReplayScratch& sx) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = lanemask_lt();
    for (int i = lane; i <= sx.hmask; i += 32) sx.hk[i] = kEmpty;
    __syncwarp();
    int nk = 0;
    for (int p0 = 0; p0 < st.np; p0 += 32) {
        const int p = p0 + lane;
        const int key = p < st.np ? st.tc[p] : -2 - lane;   // idle lanes: unique keys
        const unsigned peers = __match_any_sync(kFull, key);
        const bool lead = p < st.np && (peers & lt) == 0;
        bool is_new = false;
        unsigned h = hash_slot(key, sx.hshift);
        if (lead) {
            while (true) {
                int k = sx.hk[h];
                if (k == key) break;
                if (k == kEmpty) {
                    k = atomicCAS(sx.hk + h, kEmpty, key);   // leaders' keys differ
                    if (k == kEmpty) {
                        is_new = true;
                        break;
                    }
                }
                h = (h + 1) & sx.hmask;
            }
        }
        const unsigned nb = __ballot_sync(kFull, is_new);
        int s = 0, c0 = 0;
        if (nk + __popc(nb) > st.nscap) return false;
        if (is_new) {
            s = nk + __popc(nb & lt);
            sx.hv[h] = static_cast<unsigned char>(s);
            sx.rk[s] = key;
        } else if (lead) {
            s = sx.hv[h];
            c0 = sx.rc[s];
        }
        nk += __popc(nb);
        if (lead) sx.rc[s] = static_cast<unsigned short>(c0 + __popc(peers));
        const int src = __ffs(peers) - 1;
        s = __shfl_sync(kFull, s, src);
        c0 = __shfl_sync(kFull, c0, src);
        const int pos = c0 + __popc(peers & lt);
        // A column meets each of at most 256 steps once: pos fits a byte.
        if (p < st.np) sx.tmp[p] = static_cast<unsigned short>(s | (pos << 8));
        __syncwarp();
    }
    st.ns = nk;
    // Final numbers, columns and list starts.
    if (SORTED) {
        if (lane < 3) sx.rk[nk + lane] = INT_MAX;
        __syncwarp();
        for (int s = lane; s < nk; s += 32) {
            const int key = sx.rk[s];
            int r = 0;
            for (int j = 0; j < nk; j += 4) {
                const int4 k = *reinterpret_cast<const int4*>(sx.rk + j);
                r += (k.x < key) + (k.y < key) + (k.z < key) + (k.w < key);
            }
            sx.rid[s] = static_cast<unsigned char>(r);
            st.sc[r] = key;
            st.gst[r + 1] = sx.rc[s];
        }
    } else {
        for (int s = lane; s < nk; s += 32) {
            st.sc[s] = sx.rk[s];
            st.gst[s + 1] = sx.rc[s];
        }
    }
    __syncwarp();
    int run = 0;
    for (int s0 = 0; s0 < nk; s0 += 32) {
        const int s = s0 + lane;
        int tot;
        const int ex = wscan_excl(s < nk ? st.gst[s + 1] : 0, tot);
        const int c = s < nk ? st.gst[s + 1] : 0;
        if (s < nk) st.gst[s + 1] = static_cast<unsigned short>(run + ex + c);
        run += tot;
    }
    if (lane == 0) st.gst[0] = 0;
    __syncwarp();
    // Columns by falling count: the lanes of a round then have lists of
    // about one length.
    for (int s = lane; s < nk; s += 32) {
        const int c = st.gst[s + 1] - st.gst[s];
        int r = 0;
        for (int j = 0; j < nk; ++j) {
            const int d = st.gst[j + 1] - st.gst[j];
            r += d > c || (d == c && j < s);
        }
        st.perm[r] = static_cast<unsigned char>(s);
    }
    for (int p = lane; p < st.np; p += 32) {
        const unsigned t = sx.tmp[p];
        const int s = SORTED ? sx.rid[t & 255] : t & 255;
        st.gidx[st.gst[s] + (t >> 8)] = static_cast<unsigned short>(p);
    }
    __syncwarp();
    return true;
}

// One row's template in st (columns only).  False when the row does not fit.
template <bool SORTED, class Left>
__device__ __forceinline__ bool replay_template(const Left& L, int n, const int* __restrict__ rp,
                                                const int* __restrict__ ci, ReplayStage& st,
                                                const ReplayScratch& sx) {
    const int lane = threadIdx.x & 31;
    if (n > st.kcap) return false;
    int run = 0;
    for (int t0 = 0; t0 < n; t0 += 32) {
        const int t = t0 + lane;
        int b = 0, len = 0;
        if (t < n) {
            const int k = L.key(t);
            b = __ldg(rp + k);
            len = __ldg(rp + k + 1) - b;
        }
        int tot;
        const int o = run + wscan_excl(len, tot);
        run += tot;
        if (run > st.npcap) return false;
        if (t < n) {
            st.off[t] = static_cast<unsigned short>(o);
            sx.sb1[t] = b - o;
            for (int e = 0; e < len; ++e) st.tk[o + e] = static_cast<unsigned char>(t);
        }
    }
    if (lane == 0) st.off[n] = static_cast<unsigned short>(run);
    st.np = run;
    __syncwarp();
#pragma unroll 4
    for (int p = lane; p < run; p += 32) st.tc[p] = __ldg(ci + sx.sb1[st.tk[p]] + p);
    __syncwarp();
    if (!replay_build<SORTED>(st, sx)) return false;
    st.nst = n;
    return true;
}

// A stage of two rows at once (those of `mask`, not empty), from the
// template: key(i, t) gives step t of row i's left row (of st.nst steps; for
// a row outside the mask, the other row's, so that what is loaded through it
// is in bounds; its results are not used), val(t) stores both rows' values of
// that step to lv where they are not there yet.  Returns the rows that the
// template describes up to shift[i]; sx.prod holds their products.  U batches of
// products are loaded together.  Lanes past the end repeat the last step or
// product: loads and stores need no branches.
template <int U, bool NUM, typename TB, class Key, class Val>
__device__ __forceinline__ unsigned replay_block(unsigned mask, const ReplayStage& st, Key&& key,
                                                 Val&& val, const double2* lv,
                                                 const int* __restrict__ rp,
                                                 const int* __restrict__ ci,
                                                 const TB* __restrict__ bv,
                                                 const ReplayScratch& sx, int (&shift)[2]) {
    const int lane = threadIdx.x & 31;
    unsigned bad = ~mask;
    for (int t0 = 0; t0 < st.nst; t0 += 32) {
        const int t = min(t0 + lane, st.nst - 1);
        const int o = st.off[t], len = st.off[t + 1] - o;
        const int k0 = key(0, t), k1 = key(1, t);
        const int b0 = __ldg(rp + k0), e0 = __ldg(rp + k0 + 1);
        const int b1 = __ldg(rp + k1), e1 = __ldg(rp + k1 + 1);
        if (NUM) val(t);
        bad |= (e0 - b0 != len) | (e1 - b1 != len) << 1;
        sx.sb[t] = make_int2(b0 - o, b1 - o);
    }
    mask = ~__reduce_or_sync(kFull, bad);
    __syncwarp();
    if (!mask) return 0;
    shift[0] = shift[1] = 0;
    bad = 0;
    for (int p0 = 0; p0 < st.np; p0 += 32 * U) {
        int p[U], k[U], c0[U], c1[U];
        TB v0[U], v1[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            p[u] = min(p0 + 32 * u + lane, st.np - 1);
            k[u] = st.tk[p[u]];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int2 sb = sx.sb[k[u]];
            const int e0 = (mask & 1 ? sb.x : sb.y) + p[u];
            const int e1 = (mask & 2 ? sb.y : sb.x) + p[u];
            c0[u] = __ldg(ci + e0);
            c1[u] = __ldg(ci + e1);
            if (NUM) {
                v0[u] = __ldg(bv + e0);
                v1[u] = __ldg(bv + e1);
            }
        }
        if (p0 == 0) {
            const int tc0 = st.tc[0];
            shift[0] = __shfl_sync(kFull, c0[0], 0) - tc0;
            shift[1] = __shfl_sync(kFull, c1[0], 0) - tc0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int tc = st.tc[p[u]];
            bad |= (c0[u] - tc != shift[0]) | (c1[u] - tc != shift[1]) << 1;
            if (NUM) {
                const double2 s = lv[k[u]];
                sx.prod[p[u]] = make_double2(__dmul_rn(static_cast<double>(v0[u]), s.x),
                                             __dmul_rn(static_cast<double>(v1[u]), s.y));
            }
        }
    }
    mask &= ~__reduce_or_sync(kFull, bad);
    __syncwarp();
    return mask;
}

// The sums of column s's products in order, of both rows of a block.
__device__ __forceinline__ double2 replay_sums(const ReplayStage& st, const ReplayScratch& sx,
                                               int s) {
    const int a = st.gst[s], b = st.gst[s + 1];
    double2 x = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int j = a; j < b; ++j) {
        const double2 q = sx.prod[st.gidx[j]];
        x.x = __dadd_rn(x.x, q.x);
        x.y = __dadd_rn(x.y, q.y);
    }
    return x;
}

// Space in the booked output, taken about kReplayBook entries at a time so that
// a warp seldom waits for the cursor.
struct ReplayBook {
    unsigned long long at = 0, end = 0;
    // n entries (a CTA's rows all have the template's); -1 when the space is
    // exhausted (flagged).  Whole rows are taken, so that only a warp's last
    // handout, of at most kReplayBook entries, is not used up: with 512 for
    // rows of 86, every handout lost 82, and 200,000 rows whose space was their
    // products (17.2 M) overflowed it and were formed again with exact sizes.
    __device__ __forceinline__ long long take(const RowParams& p, int n) {
        if (end - at < static_cast<unsigned long long>(n)) {
            const unsigned long long want =
                n < kReplayBook ? kReplayBook / n * static_cast<unsigned long long>(n) : n;
            unsigned long long b = 0;
            if ((threadIdx.x & 31) == 0) b = atomicAdd(p.cursor, want);
            at = __shfl_sync(kFull, b, 0);
            end = at + want;
        }
        if (at + n > p.cap) {
            if ((threadIdx.x & 31) == 0) atomicOr(p.err, kErrBook);
            return -1;
        }
        const long long r = static_cast<long long>(at);
        at += n;
        return r;
    }
};

// The output place of a row of n entries (-1: none).
template <int MODE>
__device__ __forceinline__ long long replay_place_row(const RowParams& p, ReplayBook& book,
                                                      int row, int n) {
    if (MODE == kNumBook) {
        const long long b = book.take(p, n);
        if (b >= 0 && (threadIdx.x & 31) == 0) {
            p.row_off[row] = b;
            p.row_cnt[row] = n;
        }
        return b;
    }
    const long long b = p.c_rp[row];
    if (p.c_rp[row + 1] - b != n) {
        if ((threadIdx.x & 31) == 0) atomicOr(p.err, kErrCount);
        return -1;
    }
    return b;
}

// The last stage of a block's rows (those of `mask`).
template <int MODE, typename TO>
__device__ __forceinline__ void replay_write(unsigned mask, const ReplayStage& st,
                                             const ReplayScratch& sx, const int (&shift)[2],
                                             const RowParams& p, ReplayBook& book, int row) {
    const int lane = threadIdx.x & 31;
    if constexpr (MODE == kSymb) {
        if (lane < 2 && (mask >> lane & 1)) p.row_cnt[row + lane] = st.ns;
    } else {
        const long long base0 =
            mask & 1 ? replay_place_row<MODE>(p, book, row, st.ns) : -1;
        const long long base1 =
            mask & 2 ? replay_place_row<MODE>(p, book, row + 1, st.ns) : -1;
        int* oc = MODE == kNumBook ? p.ub_ci : p.c_ci;
        TO* ov = static_cast<TO*>(MODE == kNumBook ? p.ub_v : p.c_v);
        for (int i = lane; i < st.ns; i += 32) {
            const int s = st.perm[i];
            const double2 x = replay_sums(st, sx, s);
            const int c = st.sc[s];
            if (base0 >= 0) {
                oc[base0 + s] = c + shift[0];
                stv(ov, base0 + s, x.x);
            }
            if (base1 >= 0) {
                oc[base1 + s] = c + shift[1];
                stv(ov, base1 + s, x.y);
            }
        }
    }
}

// Mark the pair's rows of `did` as done (a batch: their table bound becomes
// 0, so that no table kernel takes them).
__device__ __forceinline__ void replay_mark(const RowParams& p, int row, unsigned did) {
    const int lane = threadIdx.x & 31;
    if (lane < 2 && (did >> lane & 1)) {
        p.done[row + lane] = 1;
        p.need_zero[row + lane] = 0;
    }
}

// The rows [c0, c1) of this CTA in pairs dealt out to its warps, block(row,
// mask, starts) for each with the rows' starts (and end) in rp loaded one
// pair ahead.  Rows that it did not do are listed, or (a batch's plan) those
// it did are marked; a warp most of whose first pairs the template did not
// describe leaves the rest untried.  DONE: only rows marked before, all of
// which it has to do (a batch's replayed numeric pass).
template <bool DONE, class Block>
__device__ __forceinline__ void replay_rows(const RowParams& p, const int* __restrict__ rp,
                                            int c0, int c1, Block&& block) {
    constexpr int kTries = 8;   // rows before a warp may give up
    const int lane = threadIdx.x & 31;
    const int step = (blockDim.x >> 5) * kReplayRows;
    int row = c0 + (threadIdx.x >> 5) * kReplayRows;
    int next[3], tried = 0, hits = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) next[i] = __ldg(rp + min(row + i, p.nrows));
    for (; row < c1; row += step) {
        if (!DONE && tried >= kTries && 2 * hits < tried) {
            if (p.done) return;
            // This warp's remaining rows: whole pairs, and perhaps a last one.
            const int pairs = (c1 - row + step - 1) / step;
            const int n = 2 * pairs - (row + (pairs - 1) * step + 1 < c1 ? 0 : 1);
            int to = 0;
            if (lane == 0) to = atomicAdd(p.left_count, n);
            to = __shfl_sync(kFull, to, 0);
            for (int i = lane; i < n; i += 32)
                p.left_rows[to + i] = row + (i >> 1) * step + (i & 1);
            return;
        }
        int at[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            at[i] = next[i];
            next[i] = __ldg(rp + min(row + step + i, p.nrows));
        }
        unsigned todo = row + 1 < c1 ? 3u : 1u;
        if (DONE) {
            todo = __ballot_sync(kFull, lane < 2 && (todo >> lane & 1) && p.done[row + lane]);
            if (!todo) continue;
        }
        const unsigned did = todo & block(row, todo, at);
        const unsigned left = todo & ~did;
        tried += __popc(todo);
        hits += __popc(did);
        if (DONE) {
            if (left && lane == 0) atomicOr(p.err, kErrCount);   // the pattern has changed
        } else if (p.done) {
            replay_mark(p, row, did);
        } else if (left) {
            int to = 0;
            if (lane == 0) to = atomicAdd(p.left_count, __popc(left));
            to = __shfl_sync(kFull, to, 0);
            if (lane < 2 && (left >> lane & 1))
                p.left_rows[to + __popc(left & ((1u << lane) - 1u))] = row + lane;
        }
        __syncwarp();
    }
}

// The rows of `mask` that have n entries, from their starts `at`; b: the
// rows' starts, for a row outside the mask the other's.
__device__ __forceinline__ unsigned replay_starts(const int (&at)[3], unsigned mask, int n,
                                                  int (&b)[2]) {
    if (at[1] - at[0] != n) mask &= ~1u;
    if (at[2] - at[1] != n) mask &= ~2u;
    b[0] = mask & 1 ? at[0] : at[1];
    b[1] = mask & 2 ? at[1] : at[0];
    return mask;
}

// The row of [c0, c1) to make the template from (warp 0): of 32 rows spread
// over the run, one of the most frequent length.
__device__ __forceinline__ int replay_pick(const int* __restrict__ rp, int c0, int c1) {
    const int lane = threadIdx.x & 31;
    const int row = c0 + static_cast<int>(static_cast<long long>(c1 - c0) * (2 * lane + 1) / 64);
    const unsigned peers = __match_any_sync(kFull, __ldg(rp + row + 1) - __ldg(rp + row));
    const unsigned most = __reduce_max_sync(kFull, __popc(peers) << 5 | (31 - lane));
    return __shfl_sync(kFull, row, 31 - static_cast<int>(most & 31));
}

// Broadcast the template's sizes from warp 0 (every thread calls it).
__device__ __forceinline__ void replay_share(ReplayStage& st, int (&box)[3]) {
    if (threadIdx.x == 0) {
        box[0] = st.np;
        box[1] = st.ns;
        box[2] = st.nst;
    }
    __syncthreads();
    st.np = box[0];
    st.ns = box[1];
    st.nst = box[2];
}

// The rows [c0, c1) of a direct product by one CTA.
template <int U, int MODE, bool DONE, typename TV, typename TO>
__device__ __forceinline__ void replay_direct(const DirectRowArgs& a, const RowParams& p, int c0,
                                              int c1) {
    constexpr bool NUM = MODE != kSymb;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int box[2][3];
    const int lane = threadIdx.x & 31;
    ReplayStage st[2];
    ReplayScratch sx;
    const TV* rv = static_cast<const TV*>(a.R.v);
    const TV* av = static_cast<const TV*>(a.A.v);
    const TV* pv = static_cast<const TV*>(a.P.v);
    replay_place(p.rcaps, NUM, blockDim.x >> 5, threadIdx.x >> 5, smem, st, &sx);
    if (threadIdx.x < 32 && c0 < c1) {
        const int row = replay_pick(a.R.rp, c0, c1);
        const int rb = __ldg(a.R.rp + row);
        const LeftG<TV> L1{a.R.ci, rv, rb};
        if (!replay_template<false>(L1, __ldg(a.R.rp + row + 1) - rb, a.A.rp, a.A.ci, st[0], sx) ||
            !replay_template<true>(LeftR{st[0].sc}, st[0].ns, a.P.rp, a.P.ci, st[1], sx))
            st[0].nst = -1;
    }
    replay_share(st[0], box[0]);
    replay_share(st[1], box[1]);
    ReplayBook book;
    replay_rows<DONE>(p, a.R.rp, c0, c1, [&](int row, unsigned mask, const int (&at)[3]) -> unsigned {
        if (st[0].nst < 0) return 0;
        int rb[2], sh1[2], sh2[2];
        mask = replay_starts(at, mask, st[0].nst, rb);
        if (!mask) return 0;
        mask = replay_block<U, NUM>(
            mask, st[0], [&](int i, int t) { return __ldg(a.R.ci + rb[i] + t); },
            [&](int t) { sx.ss[t] = make_double2(ldv(rv, rb[0] + t), ldv(rv, rb[1] + t)); },
            sx.ss, a.A.rp, a.A.ci, av, sx, sh1);
        if (!mask) return 0;
        if (NUM) {
            for (int i = lane; i < st[0].ns; i += 32) {
                const int s = st[0].perm[i];
                sx.rav[s] = replay_sums(st[0], sx, s);
            }
            __syncwarp();
        }
        if (!(mask & 1)) sh1[0] = sh1[1];
        if (!(mask & 2)) sh1[1] = sh1[0];
        mask = replay_block<U, NUM>(
            mask, st[1], [&](int i, int t) { return st[0].sc[t] + sh1[i]; }, [](int) {}, sx.rav,
            a.P.rp, a.P.ci, pv, sx, sh2);
        if (mask) {
            replay_write<MODE, TO>(mask, st[1], sx, sh2, p, book, row);
            if (MODE != kNumExact && p.row_cnt1 && lane < 2 && (mask >> lane & 1))
                p.row_cnt1[row + lane] = st[0].ns;
        }
        return mask;
    });
}

template <int U, int MODE, typename TV, typename TO>
__global__ void __launch_bounds__(128, replay_ctas(U)) k_direct_replay(DirectRowArgs a, RowParams p) {
    const int c0 = static_cast<int>(static_cast<long long>(p.nrows) * blockIdx.x / gridDim.x);
    const int c1 =
        static_cast<int>(static_cast<long long>(p.nrows) * (blockIdx.x + 1) / gridDim.x);
    replay_direct<U, MODE, false, TV, TO>(a, p, c0, c1);
}

// Runs of rows of a batch's direct products: CTA c takes rows [y, z) of
// product chunks[c].x.
template <int U, int MODE, typename TV, typename TO>
__global__ void __launch_bounds__(128, replay_ctas(U))
    k_batch_replay(const BItem* __restrict__ items, const int4* __restrict__ chunks,
                   BatchRowParams b, BatchReplay r) {
    const int4 ch = chunks[blockIdx.x];
    const BItem* I = items + ch.x;
    const long long g = I->row_base;
    const DirectRowArgs a{I->X, I->Y, I->Z};
    RowParams p{};
    p.nrows = I->M;
    p.c_vt = r.to;
    p.err = b.err;
    p.rcaps = r.caps;
    p.done = r.done + g;
    if (MODE == kNumExact) {
        p.c_rp = b.c_rp + g;
        p.c_ci = b.c_ci;
        p.c_v = b.c_v;
    } else {
        p.need_zero = r.need_zero + g;
        p.row_cnt = b.cnt2 + g;
        p.row_cnt1 = b.cnt1 + g;
        if (MODE == kNumBook) {
            p.cursor = b.cursor;
            p.cap = b.cap;
            p.row_off = b.row_off + g;
            p.ub_ci = b.ub_ci;
            p.ub_v = b.ub_v;
        }
    }
    replay_direct<U, MODE, MODE == kNumExact, TV, TO>(a, p, ch.y, ch.z);
}

template <int U, int MODE, typename TV, typename TO>
__global__ void __launch_bounds__(128, replay_ctas(U)) k_pair_replay(PairRowArgs a, RowParams p) {
    constexpr bool NUM = MODE != kSymb;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int box[3];
    ReplayStage st[2];
    ReplayScratch sx;
    const TV* avals = static_cast<const TV*>(a.A.v);
    const TV* bvals = static_cast<const TV*>(a.B.v);
    const int c0 = static_cast<int>(static_cast<long long>(p.nrows) * blockIdx.x / gridDim.x);
    const int c1 =
        static_cast<int>(static_cast<long long>(p.nrows) * (blockIdx.x + 1) / gridDim.x);
    replay_place(p.rcaps, NUM, blockDim.x >> 5, threadIdx.x >> 5, smem, st, &sx);
    if (threadIdx.x < 32 && c0 < c1) {
        const int row = replay_pick(a.A.rp, c0, c1);
        const int ab = __ldg(a.A.rp + row);
        const LeftG<TV> L{a.A.ci, avals, ab};
        if (!replay_template<true>(L, __ldg(a.A.rp + row + 1) - ab, a.B.rp, a.B.ci, st[0], sx))
            st[0].nst = -1;
    }
    replay_share(st[0], box);
    ReplayBook book;
    replay_rows<false>(p, a.A.rp, c0, c1, [&](int row, unsigned mask, const int (&at)[3]) -> unsigned {
        if (st[0].nst < 0) return 0;
        int ab[2], sh[2];
        mask = replay_starts(at, mask, st[0].nst, ab);
        if (!mask) return 0;
        mask = replay_block<U, NUM>(
            mask, st[0], [&](int i, int t) { return __ldg(a.A.ci + ab[i] + t); },
            [&](int t) { sx.ss[t] = make_double2(ldv(avals, ab[0] + t), ldv(avals, ab[1] + t)); },
            sx.ss, a.B.rp, a.B.ci, bvals, sx, sh);
        if (mask) replay_write<MODE, TO>(mask, st[0], sx, sh, p, book, row);
        return mask;
    });
}

}  // namespace sp3mm
