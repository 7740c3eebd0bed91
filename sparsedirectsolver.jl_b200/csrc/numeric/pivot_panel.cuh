// Wide LDLT (Bunch-Kaufman) and LU (threshold) fronts of one-member plans, 32 columns at a time.
//
// A front's leader (one CTA, or one cluster whose CTAs share the rows) holds the current block of at most
// 32 columns in registers, one row per thread, and runs the pivot steps there: per step one exchange of
// the column's maxima over distributed shared memory (the block's own rows are held by every CTA), and the
// rank-1 (rank-2) update of the block's columns in registers. The rest of the front takes the whole block
// at once: the block's rows are solved against its unit triangle (T1), then every entry takes the block's
// products one after another (T2), by the leader and the front's helper CTAs.
//
// What bounds it: the chain of pivot steps, 1.6 us a column with everything (lap3d 40^3 "S": 8.9 ms over the
// 5477 columns of the tree's wide fronts, level by level; 40^3 LU 10.4 ms; with the loop's short loops unrolled 9.7
// and 11.0 ms; with every pivot row sent by the CTA that holds it as well 10.8 and 12.3 ms; with the statistics in
// every thread and D written inside the chain as well 12.2 ms "S"; with plain remote stores and a cluster barrier per
// step 14.4 and 14.1 ms; the cooperative kernel's two group barriers a column in global memory 58.8 and 71.3 ms). The
// updates run at a few percent of the FP64 rate; T2's tiles double-buffered cost LU 14.7 ms (registers).
//
// Every entry receives the products of ldlt_front_steps / lu_front_steps (front_factor.cuh) in the same
// order, each product and difference rounded on its own, and every pivot decision sees the same values, so
// pivots, D and panels are those of the one-CTA kernel bit for bit.
//
// A Bunch-Kaufman partner may lie outside the block. Its column is then brought up to date by itself: the block's
// eliminated rows are solved against their triangle in that column, and every row takes their products (pp_bring).
// If it becomes a pivot, it takes the place of the block's column, whose values from before the block go where it
// was, for the block's later products. (Ending the block at every such pivot made a dense random front of 2400
// columns 48.7 ms and one whose partners are all far 39.9 ms, against 35.9 and 31.7 ms of the cooperative kernel.)
// The search over all diagonals after a rejected choice needs the whole front up to date: it ends the block, unless
// the rejected one is its first.
#pragma once
#include <stdint.h>

#include "common.cuh"
#include "front_factor.cuh"
#include "kernels.cuh"
#include "pivot.cuh"

namespace sds {

constexpr int PP_WARPS = PP_THREADS / 32;
constexpr int PP_TR = 128, PP_TC = 64;   // rows and columns of an update tile: 4 x 4 entries per thread
static_assert(PP_TR * PP_TC == 16 * PP_THREADS, "an update tile holds 16 entries per thread");

template <typename T>
struct PanelSmem {
    T prow[PP_NB][PP_NB + 2];                              // the pivot rows as they were eliminated, entry e at
                                                           // e + 1: entries (1, 2), (3, 4), ... are aligned pairs
    unsigned long long mbar[2];                            // the leader's exchanges, by turns
    unsigned hi[2][PP_MAXC * PP_WARPS];                    // per warp: an upper bound of the column's entries
    unsigned long long lam[PP_MAXC * PP_WARPS];            // per warp: the column's largest entry above row w
    unsigned long long mx[PP_MAXC * PP_WARPS];             // ... and of all rows (NaN wins)
    int ridx[PP_MAXC * PP_WARPS];
    unsigned long long sg[PP_MAXC * PP_WARPS], m1[PP_MAXC * PP_WARPS], m2[PP_MAXC * PP_WARPS];
    T sc[4];                                               // F[r, r], F[k, r], F[r, k]
    int plp, nbd, ok;
    int gate;                                              // the leader's first CTA: its warps go into the search together
    int fail;                                              // a warp's wait in this block gave up
    int dead;                                              // ... one of the cluster's; every CTA's word is set
    PanelLimit limit;
    unsigned epoch, xn;
    int sel[2];
    int kind[PP_NB];
    double tdk[PP_NB], tee[PP_NB];
    int st[NSTAT];                                         // the statistics (thread 0 of the leader's first CTA)
    double red[PP_WARPS];
    int redi[PP_WARPS];
    PanelHdr<T> hdr;                                       // T1 / T2: the block's header; "S", between them: the pivot rows'
                                                           // multipliers and first places that pp_bring needs
    union {
        T L[PP_NB][PP_THREADS];                            // the block: the rows' multipliers
        struct {
            T Rs[PP_NB][PP_TR];                            // T2: a tile's operands
            T Cs[PP_NB][PP_TC];
        };
    };
};

// --- keys: |v| as an integer in the order of the values; NaN above infinity -------------------------------------
__device__ __forceinline__ unsigned long long pp_key(double v) {
    return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}
__device__ __forceinline__ unsigned long long pp_key(float v) { return __float_as_uint(v) & 0x7fffffffu; }
template <typename T>
__device__ __forceinline__ double pp_val(unsigned long long k) {
    if constexpr (sizeof(T) == 8) return __longlong_as_double((long long)k);
    else return (double)__uint_as_float((unsigned)k);
}
template <typename T>
__device__ __forceinline__ unsigned long long pp_inf() {
    return sizeof(T) == 8 ? 0x7ff0000000000000ull : 0x7f800000ull;
}
template <typename T>
__device__ __forceinline__ unsigned long long pp_warp_max(unsigned long long k) {
    if constexpr (sizeof(T) == 8) {
        const unsigned hi = (unsigned)(k >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
        const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)k : 0u);
        return ((unsigned long long)mh << 32) | ml;
    } else {
        return __reduce_max_sync(0xffffffffu, (unsigned)k);
    }
}
// the part of a key that one 32-bit reduction takes, and a value no smaller than any with that part (NaN
// for infinities and NaN)
__device__ __forceinline__ unsigned pp_hi(double v) { return (unsigned)(pp_key(v) >> 32); }
__device__ __forceinline__ unsigned pp_hi(float v) { return (unsigned)pp_key(v); }
template <typename T>
__device__ __forceinline__ double pp_bound(unsigned h) {
    if constexpr (sizeof(T) == 8)
        return __longlong_as_double((long long)((unsigned long long)(h >= 0x7ff00000u ? 0x7ff80000u : h + 1u) << 32));
    else return h >= 0x7f800000u ? __longlong_as_double(0x7ff8000000000000ll) : (double)__uint_as_float(h);
}
// the largest key and, among equal ones, the smallest index; a zero key has no index (-1)
template <typename T>
__device__ __forceinline__ unsigned long long pp_warp_argmax(unsigned long long k, int& idx) {
    const unsigned long long m = pp_warp_max<T>(k);
    const unsigned i = __reduce_min_sync(0xffffffffu, k == m ? (unsigned)idx : 0xffffffffu);
    idx = m == 0 ? -1 : (int)i;
    return m;
}

// --- a front as its CTAs see it -----------------------------------------------------------------------------------
template <typename T, bool GEN>
struct PanelFront {
    T* P;
    T* U;
    int f, w, c0;
    double* dd;
    double* ee;
    int* lp;
    signed char* kd;
    PanelHdr<T>* hdr;
    T* us;             // the block's rows right of it, solved and unscaled: us[t f + c]
    int C, rank;       // the leader's CTAs and this CTA's rank among them
    int gs, grank;     // the front's CTAs and this CTA's rank among them
    int par;           // the block's parity
    unsigned xn;       // exchanges of the leader's CTAs so far (the same in each)
    unsigned int* bar;
    unsigned int* epoch;   // shared memory
    const PanelLimit* limit;   // shared memory
    int* ok;           // shared memory: the front's barriers have held so far
    int* dead;         // shared memory, set in every CTA of the cluster
    // F[i, j], i or j < w
    __device__ T& at(int i, int j) const {
        if (!GEN || (i >= j && j < w)) return P[i + (int64_t)j * f];
        return U[j + (int64_t)i * f];
    }
    __device__ double get(int i, int j) const { return (double)at(i, j); }
    __device__ int scan_rows() const { return f; }
    __device__ double part_max(int, int, int) const { return 0.0; }
};

// the leader's CTAs meet; their writes before it (shared, distributed shared and global) are visible after
template <typename T, bool GEN>
__device__ __forceinline__ void pp_sync(const PanelFront<T, GEN>& F) {
    if (F.C > 1) pp_cluster_barrier();
    else __syncthreads();
}

// every CTA of the front meets; false once a bounded wait has given up (the same for the whole CTA)
template <typename T, bool GEN>
__device__ __forceinline__ bool pp_group_sync(PanelFront<T, GEN>& F) {
    if (F.gs > F.C) {
        pp_group_barrier(F.bar, *F.epoch, F.gs, *F.limit, F.ok);
        return *F.ok != 0;
    }
    pp_sync(F);
    return true;
}
// This CTA has given up: the cluster's CTAs learn of it at their next cluster barrier
template <typename T, bool GEN>
__device__ __forceinline__ void pp_give_up(const PanelFront<T, GEN>& F) {
    if (threadIdx.x == 0)
        for (int q = 0; q < F.C; ++q) pp_remote_set(F.dead, q, 1);
}

template <typename T>
__device__ __forceinline__ T pp_pick(const T (&a)[PP_NB], int x) {
    T v = a[0];
#pragma unroll
    for (int e = 1; e < PP_NB; ++e)
        if (e == x) v = a[e];
    return v;
}

// --- exchanges of the leader's CTAs ---------------------------------------------------------------------------------
// Every leader CTA sends what the others need with asynchronous stores that count into the receiver's
// mbarrier, and waits for its own. (Stores, then a cluster barrier: 0.25 us for the barrier alone, 0.7 us with
// the maxima and the row, whose completion the barrier's release waits for.)
// Two mbarriers take turns, so an exchange's bytes must not arrive while a receiver still waits for the one
// before the last. Every warp of every CTA therefore has a part in every exchange, sent when it has closed the
// last: whoever closes an exchange knows that all the others have closed the one before, and with it that all
// its bytes have arrived everywhere. An exchange of one sender alone (a row, a choice) takes join() of the rest.
// Only the warps that hold rows (or the copies, below) take part. One CTA alone meets at a barrier of those warps instead.
template <typename T, bool GEN>
struct PanelX {
    PanelSmem<T>& S;
    const int C, rank, nw;
    int b;
    unsigned xn;
    __device__ PanelX(PanelSmem<T>& S_, int C_, int rank_, int nw_, unsigned xn_)
        : S(S_), C(C_), rank(rank_), nw(nw_), b(0), xn(xn_) {}
    // opens the next exchange, of `bytes` bytes into each CTA
    __device__ __forceinline__ void open(int bytes) {
        b = xn & 1;
        if (C > 1 && threadIdx.x == 0) pp_x_arm(&S.mbar[b], bytes);
    }
    template <typename V>
    __device__ __forceinline__ void put(V* p, int q, V v) const {   // into CTA q's copy of *p
        if (C > 1) pp_x_store(p, q, v, &S.mbar[b]);
        else *p = v;
    }
    // This lane's view: false, its wait gave up. A warp leaves the block when a lane's did; nothing that was
    // exchanged may be used then. The others wait in vain for its next part and follow.
    __device__ __forceinline__ bool close_lane() {
        bool ok = true;
        if (C > 1) ok = pp_x_wait(&S.mbar[b], (xn >> 1) & 1, S.limit);
        else pp_warps_barrier(nw * 32);
        xn++;
        return ok;
    }
    __device__ __forceinline__ bool close() { return __all_sync(0xffffffffu, close_lane()); }
    // the warp's part in an exchange to which it has nothing to say, and the bytes of all of them
    __device__ __forceinline__ void join() const {
        const int lane = threadIdx.x & 31;
        if (C > 1 && lane < C) put(&S.hi[b][rank * nw + (threadIdx.x >> 5)], lane, 0u);
    }
    __device__ int join_bytes() const { return C * nw * 4; }
    // the warps meet: what they wrote to global memory is visible
    __device__ __forceinline__ bool meet() {
        __threadfence();
        __syncwarp();
        __threadfence();
        open(join_bytes());
        join();
        const bool ok = close();
        __threadfence();
        return ok;
    }
    // The next exchange, of maxima, with row `pos` from the CTA's own copy: the warp that holds it (`copy`) writes
    // the row and then opens the exchange, so whoever has waited for the maxima sees the row. Whole warps call it.
    __device__ __forceinline__ void open_with_copy(bool copy, const T (&a)[PP_NB], int rp, int pos, int t, int left) {
        b = xn & 1;
        if (!copy) return;
        if (rp == pos) write_row(a, S.prow[t], left);
        __syncwarp();
        if ((threadIdx.x & 31) == 0) pp_x_arm(&S.mbar[b], C * nw * 4);
    }
    __device__ static __forceinline__ void write_row(const T (&a)[PP_NB], T* row, int left) {
        row[1] = a[0];
#pragma unroll
        for (int g = 0; g < PP_NB; g += 8)
            if (g + 1 < left) {
#pragma unroll
                for (int e = g + 1; e < g + 9 && e + 1 < PP_NB; e += 2) pp_store2(row + e + 1, a[e], a[e + 1]);
            }
        row[PP_NB] = a[PP_NB - 1];
    }
    // bytes of a pivot row with `left` live entries, as whole pairs
    __device__ static int row_bytes(int left) { return (left + 2) / 2 * 2 * (int)sizeof(T); }
    // The thread that holds row `pos` writes its `left` live entries to prow[t], and its warp sends them to
    // every CTA, a pair per store. Whole warps call it, inside an exchange.
    __device__ __forceinline__ void row(const T (&a)[PP_NB], int rp, int pos, int t, int left) const {
        if (__ballot_sync(0xffffffffu, rp == pos) == 0) return;
        T* row = S.prow[t];
        if (rp == pos) write_row(a, row, left);
        __syncwarp();
        if (C > 1) {
            const int lane = threadIdx.x & 31, per = 32 / C, q = lane / per, ch = (left + 2) / 2;
#pragma unroll 1
            for (int c = lane % per; c < ch; c += per) pp_x_store2(row + 2 * c, q, row[2 * c], row[2 * c + 1], &S.mbar[b]);
        }
    }
};

// the warps of a CTA that hold rows, as a team (pivot.cuh)
struct PanelTeam {
    int rank, size;
    double* red;
    int* redi;
    __device__ double reduce_jmax(double v) const {
        v = warp_jmax(v);
        pp_warps_barrier(size);
        if ((rank & 31) == 0) red[rank >> 5] = v;
        pp_warps_barrier(size);
        double r = red[0];
#pragma unroll 1
        for (int w = 1; w < (size >> 5); ++w) r = jmax(r, red[w]);
        return r;
    }
    __device__ void reduce_argmax(double& v, int& idx) const {
        warp_argmax(v, idx);
        pp_warps_barrier(size);
        if ((rank & 31) == 0) {
            red[rank >> 5] = v;
            redi[rank >> 5] = idx;
        }
        pp_warps_barrier(size);
        v = red[0];
        idx = redi[0];
#pragma unroll 1
        for (int w = 1; w < (size >> 5); ++w)
            if (red[w] > v || (red[w] == v && redi[w] >= 0 && (idx < 0 || redi[w] < idx))) {
                v = red[w];
                idx = redi[w];
            }
    }
};

// The reference's best_1x1 and what follows a rejected choice (bc, br), by one CTA over the whole, up to date
// front: the acceptable diagonal of largest magnitude, first on ties, tried in that order
template <typename T, bool GEN>
__device__ void pp_search(const PanelFront<T, GEN>& F, PanelSmem<T>& S, int nw, int k, int pivot, double u, double eps, int bc,
                          int br, int& c_out, int& r_out) {
    const PanelTeam tm{(int)threadIdx.x, nw * 32, S.red, S.redi};
    r_out = -1;
    double la = -1.0;      // the last candidate tried; -1: none yet
    int lj = -1;
    while (true) {
        double a = -1.0;
        int j = -1;
#pragma unroll 1
        for (int i = k + tm.rank; i < F.w; i += tm.size) {
            const double x = fabs(F.get(i, i));
            if (!(x >= eps)) continue;
            if (lj >= 0 && !(x < la || (x == la && i > lj))) continue;
            if (x > a) { a = x; j = i; }
        }
        tm.reduce_argmax(a, j);
        if (j < 0) break;
        if (threshold_ok(F, j, k, u, a, tm)) { c_out = j; return; }
        la = a;
        lj = j;
    }
    if (pivot == PIVOT_DIAGONAL) {
        const double a0 = fabs(F.get(k, k));
        double a = -1.0;
        int j = -1;
#pragma unroll 1
        for (int i = k + 1 + tm.rank; i < F.w; i += tm.size) {
            const double x = fabs(F.get(i, i));
            if (x > a) { a = x; j = i; }
        }
        tm.reduce_argmax(a, j);
        const int big = (j >= 0 && a > a0) ? j : k;
        c_out = fabs(F.get(big, big)) >= eps ? big : k;
        return;
    }
    if (br >= 0 && nonsingular_2x2_w(F, k, br, eps)) r_out = br;
    c_out = bc;
}

// The row's up-to-date entry of column r, outside the block, behind the block's first j steps (of which `firsts` begin
// a 2x2 pair); 0 for finished rows. Pivot rows sent .. j - 1 send their multipliers first (exchange xn). Every warp
// solves the column's entries of the pivot rows for itself, row t by lane t, while its rows take the products. A
// call, so that the step's loop stays small.
template <typename T>
struct PanelEntry {
    T v;
    int ok;   // 0: a wait gave up
};
template <typename T>
__device__ __noinline__ PanelEntry<T> pp_bring(PanelSmem<T>& S, const T* column, int C, int rank, int nw, unsigned xn, int k0, int j,
                                               int sent, unsigned firsts, int rp, int src, int spare) {
    const int tid = threadIdx.x, lane = tid & 31;
    T v = rp >= k0 + j ? __ldcg(column + src) : T(0);
    if (j == 0) return {v, 1};
    if (sent < j) {
        PanelX<T, false> X(S, C, rank, nw, xn);
        X.open(X.join_bytes() + (j - sent) * 4 + (j * (j - 1) - sent * (sent - 1)) / 2 * (int)sizeof(T));
        X.join();
        for (int t = sent; t < j; ++t) {
            const unsigned own = __ballot_sync(0xffffffffu, rp == k0 + t && !spare);
            if (own == 0) continue;
            const int o = __ffs(own) - 1, at = __shfl_sync(0xffffffffu, src, o);
            if (lane < C) X.put(&S.hdr.rowmap[t], lane, at);
            for (int i = lane; i < C * t; i += 32) X.put(&S.hdr.lt[i % t][t], i / t, S.L[i % t][tid - lane + o]);
        }
        if (!X.close()) return {T(0), 0};
    }
    T g = lane < j ? __ldcg(column + S.hdr.rowmap[lane]) : T(0);
    for (int s = 0; s < j;) {
        const T u = __shfl_sync(0xffffffffu, g, s);
        if (firsts >> s & 1) {
            const T u1 = __shfl_sync(0xffffffffu, g, s + 1);
            if (lane > s + 1) g -= S.hdr.lt[s][lane] * u + S.hdr.lt[s + 1][lane] * u1;
            if (rp >= k0 + j) v -= S.L[s][tid] * u + S.L[s + 1][tid] * u1;
            s += 2;
        } else {
            if (lane > s) g -= S.hdr.lt[s][lane] * u;
            if (rp >= k0 + j) v -= S.L[s][tid] * u;
            s += 1;
        }
    }
    return {v, 1};
}

struct PanelPivot {
    int pivot, lu_pivot;
    double u, eps;
    const int8_t* psign;
    const int32_t* perm;
};

// The pivot steps of the block that starts at column k0, by the leader's CTAs. Returns k1, the first column
// that is left, or -1 (the whole CTA) after a wait that gave up.
//
// A step is a chain of latencies, not of work: the maxima to the other CTAs, the decision,
// a division, the update of up to 31 columns. The loop over the steps has to stay small for the instruction caches:
// short loops in it are not unrolled (pivot launches 9.7 -> 8.9 ms lap3d 40^3 "S", 16.6 -> 15.6 KKT 80 x 75, 11.0 ->
// 10.4 40^3 LU).
template <typename T, int STRUCT>
__device__ int pp_block(PanelFront<T, STRUCT == STRUCT_G>& F, PanelSmem<T>& S, const PanelPivot& pv, int k0) {
    constexpr bool GEN = STRUCT == STRUCT_G;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int f = F.f, w = F.w, C = F.C, rank = F.rank;
    const int nb = min(PP_NB, w - k0), kend = k0 + nb;
    // rows k0 .. f - 1 in one contiguous, warp-aligned chunk per CTA
    const int chunk = ((f - k0 + C - 1) / C + 31) & ~31;
    const int rows = chunk >> 5;
    const int orig = tid < chunk && k0 + rank * chunk + tid < f ? k0 + rank * chunk + tid : -1;
    // Every leader CTA has a copy of the block's rows, in one warp more, and updates them like its own: the pivot
    // row of a step never travels unless it comes from outside the block. The warp takes part in every exchange
    // (with zeros). Blocks of more than 15 warps a CTA go without.
    const bool copies = C > 1 && rows < PP_WARPS, spare = copies && warp == rows;
    const int nw = rows + copies, nparts = C * nw;
    const int src = spare ? (k0 + lane < f ? k0 + lane : -1) : orig;
    int rp = src;                       // the row's place; a finished row keeps its own (<= k)
    T a[PP_NB];                         // the row's entries of columns k, k + 1, ...: the columns move down by one
                                        // with every eliminated one, so that no index depends on k
    const double alpha = (1.0 + sqrt(17.0)) / 8.0;
#pragma unroll
    for (int e = 0; e < PP_NB; ++e) a[e] = (src >= 0 && e < nb) ? F.at(src, k0 + e) : T(0);
    const int mylp = (orig >= 0 && orig < w) ? F.lp[orig] : 0;
    // the next block's counters: the last one's, which every CTA has read, and the meetings of the group behind this
    // block come before anyone counts in them
    if (rank == 0 && tid == 0) F.hdr->ndisp[F.par ^ 1] = F.hdr->moved[F.par ^ 1] = 0;
    if (warp < nw) {
        PanelX<T, GEN> X(S, C, rank, nw, F.xn);
        int j = 0;
        bool gave_up = false;
        // "S", lane e: where in the block column k0 + e was when it began; step e begins a 2x2 pair; every CTA has
        // pivot row e's multipliers (for pp_bring: in one register, of which the steps without it need none)
        constexpr int FIRST = PP_NB, SENT = 2 * PP_NB;
        int from = lane;
        while (j < nb) {
            const int k = k0 + j, left = nb - j;   // columns k .. kend - 1
            // a bound of the column below row k, and row k itself, to every leader CTA
            if (copies) X.open_with_copy(spare, a, rp, k, j, left);
            else X.open(nparts * 4 + X.row_bytes(left));
            unsigned h = __reduce_max_sync(0xffffffffu, rp > k && !spare ? pp_hi(a[0]) : 0u);
            if (lane < C) X.put(&S.hi[X.b][rank * nw + warp], lane, h);
            if (!copies) X.row(a, rp, k, j, left);
            // (no entry's part is all ones: its sign is cleared)
            h = X.close_lane() ? 0u : 0xffffffffu;
#pragma unroll 1
            for (int i = lane; i < nparts; i += 32) h = max(h, S.hi[X.b][i]);
            h = __reduce_max_sync(0xffffffffu, h);
            if (h == 0xffffffffu) { gave_up = true; break; }
            const double bound = pp_bound<T>(h);
            const double fkk = (double)S.prow[j][1], akk = fabs(fkk);   // read once: an interchange overwrites the row
            // The bound alone accepts most pivots (every test grows with the maxima). Else the exact maxima:
            // lambda = max over the rows k < i < w with its first row r, mall = max over all rows i > k (NaN wins).
            bool fast;
            if (GEN) fast = !pv.lu_pivot || (akk >= pv.u * bound && akk >= pv.u * akk);
            else if (pv.pivot == PIVOT_NONE) fast = true;
            else fast = akk >= pv.eps && akk >= pv.u * bound && (pv.pivot == PIVOT_DIAGONAL || akk >= alpha * bound);
            int c = k, r2 = -1;
            bool searched = false;
            T v;                                         // "S": the row's entry of the partner's column
            if (!fast) {
                const unsigned long long key = rp > k ? pp_key(a[0]) : 0ull;
                const unsigned long long mkey = pp_warp_max<T>(key);
                int ri = rp;
                const unsigned long long lkey =
                    pp_warp_argmax<T>(rp > k && rp < w && key <= pp_inf<T>() ? key : 0ull, ri);
                X.open(nparts * 20);
                if (lane < C) {
                    const int at = rank * nw + warp;
                    X.put(&S.lam[at], lane, lkey);
                    X.put(&S.mx[at], lane, mkey);
                    X.put(&S.ridx[at], lane, ri);
                }
                if (!X.close()) { gave_up = true; break; }
                unsigned long long lk = 0, mk = 0;
                int r = 0x7fffffff;
#pragma unroll 1
                for (int i = lane; i < nparts; i += 32) {
                    const unsigned long long l = S.lam[i], m = S.mx[i];
                    const int x = S.ridx[i];
                    if (l > lk || (l == lk && l != 0 && x < r)) { lk = l; r = x; }
                    if (m > mk) mk = m;
                }
                lk = pp_warp_argmax<T>(lk, r);
                const double lambda = pp_val<T>(lk), mall = pp_val<T>(pp_warp_max<T>(mk));
                if (GEN) {
                    if (!(akk >= pv.u * jmax(mall, akk)) && r >= 0 && lambda > akk) c = r;
                } else {
                    bool acc;
                    int bc = k, br = -1;
                    v = T(0);
                    if (pv.pivot == PIVOT_DIAGONAL || r < 0 || akk >= alpha * lambda) {
                        acc = akk >= pv.eps && akk >= pv.u * mall;
                    } else {
                        // column r: its maxima, those of column k without row r, and the corner entries
                        if (r >= kend) {
                            const unsigned firsts = __ballot_sync(0xffffffffu, from & FIRST);
                            const int sent = __popc(__ballot_sync(0xffffffffu, from & SENT));
                            const PanelEntry<T> e = pp_bring<T>(S, &F.at(0, r), C, rank, nw, X.xn, k0, j, sent, firsts, rp, src, spare);
                            X.xn += sent < j;
                            if (lane < j) from |= SENT;
                            if (!e.ok) { gave_up = true; break; }
                            v = e.v;
                        } else if (rp >= k) {
                            v = pp_pick(a, r - k);
                        }
                        const unsigned long long kv = rp >= k && rp != r ? pp_key(v) : 0ull;
                        unsigned long long s1 = pp_warp_max<T>(rp < w ? kv : 0ull);
                        unsigned long long s2 = pp_warp_max<T>(rp != k ? kv : 0ull);
                        unsigned long long s3 = pp_warp_max<T>(rp > k && rp != r ? pp_key(a[0]) : 0ull);
                        X.open(nparts * 24 + 3 * (int)sizeof(T));
                        if (lane < C) {
                            const int at = rank * nw + warp;
                            X.put(&S.sg[at], lane, s1);
                            X.put(&S.m2[at], lane, s2);
                            X.put(&S.m1[at], lane, s3);
                        }
                        if (rp == r && !spare)
#pragma unroll 1
                            for (int q = 0; q < C; ++q) {
                                X.put(&S.sc[0], q, v);
                                X.put(&S.sc[2], q, a[0]);
                            }
                        if (rp == k && !spare)
#pragma unroll 1
                            for (int q = 0; q < C; ++q) X.put(&S.sc[1], q, v);
                        if (!X.close()) { gave_up = true; break; }
                        s1 = s2 = s3 = 0;
#pragma unroll 1
                        for (int i = lane; i < nparts; i += 32) {
                            if (S.sg[i] > s1) s1 = S.sg[i];
                            if (S.m2[i] > s2) s2 = S.m2[i];
                            if (S.m1[i] > s3) s3 = S.m1[i];
                        }
                        const double sigma = pp_val<T>(pp_warp_max<T>(s1)), m2 = pp_val<T>(pp_warp_max<T>(s2)),
                                     m1 = pp_val<T>(pp_warp_max<T>(s3));
                        const double frr = (double)S.sc[0], fkr = (double)S.sc[1], frk = (double)S.sc[2];
                        if (akk * sigma >= alpha * lambda * lambda) {
                            acc = akk >= pv.eps && akk >= pv.u * mall;
                        } else if (fabs(frr) >= alpha * sigma) {
                            bc = r;
                            acc = fabs(frr) >= pv.eps && fabs(frr) >= pv.u * jmax(m2, fabs(fkr));
                        } else {
                            br = r;
                            const double det = fkk * frr - fkr * frk;
                            const double big = jmax(jmax(fabs(fkk), fabs(frk)), fabs(frr));
                            acc = det != 0.0 && isfinite(det) && big >= pv.eps;
                            if (acc) {
                                const double e11 = fabs(frr / det), e12 = fabs(fkr / det), e21 = fabs(frk / det),
                                             e22 = fabs(fkk / det);
                                acc = pv.u * (e11 * m1 + e21 * m2) <= 1.0 && pv.u * (e12 * m1 + e22 * m2) <= 1.0;
                            }
                        }
                    }
                    c = bc;
                    r2 = br;
                    if (acc && br >= 0 && left < 2) break;   // a pair needs two of the block's columns
                    if (!acc) {
                        searched = true;
                        if (j > 0) break;                // the search needs the whole front up to date
                        X.open(X.join_bytes() + 8);
                        if (rank == 0) {
                            // the search has barriers of the CTA's warps: all of them, or none
                            bool in = C == 1;
                            if (C > 1 && lane == 0) in = pp_gate(&S.gate, nw, S.limit);
                            if (!__any_sync(0xffffffffu, in)) { gave_up = true; break; }
                            int cs = k, rs = -1;
                            pp_search(F, S, nw, k, pv.pivot, pv.u, pv.eps, bc, br, cs, rs);
                            if (tid == 0)
#pragma unroll 1
                                for (int q = 0; q < C; ++q) {
                                    X.put(&S.sel[0], q, cs);
                                    X.put(&S.sel[1], q, rs);
                                }
                        }
                        X.join();                        // behind the search: its reads are done when this closes
                        if (!X.close()) { gave_up = true; break; }
                        c = S.sel[0];
                        r2 = S.sel[1];
                    }
                }
                const int p = r2 < 0 ? k : k + 1, q = r2 < 0 ? c : r2;
                if (p != q || r2 >= 0) {
                    // (the last exchange is closed: everyone has read row k and the columns that change below)
                    if (p != q && q < kend) {            // "S" inside the block: columns in registers; rows by place
                        if (!GEN && rp >= k) {
                            const int y = q - k;
                            const T vp = p == k ? a[0] : a[1], vq = pp_pick(a, y);
                            if (p == k) a[0] = vq;
                            else a[1] = vq;
#pragma unroll
                            for (int e = 1; e < PP_NB; ++e)
                                if (e == y) a[e] = vp;
                        }
                        if (rp == p) rp = q;
                        else if (rp == q) rp = p;
                        if (!GEN) {
                            const int fp = __shfl_sync(0xffffffffu, from, p - k0), fq = __shfl_sync(0xffffffffu, from, q - k0);
                            if (lane == p - k0) from = fq;   // (neither is eliminated: no other bits)
                            else if (lane == q - k0) from = fp;
                        }
                    } else if (p != q && GEN) {          // row interchange: rows change places, their data stay
                        if (rp == p) rp = q;
                        else if (rp == q) rp = p;
                    } else if (p != q) {                 // outside it: v, and the old column's first values for later
                        if (searched) {                  // (j = 0: every column is up to date)
                            v = rp >= k ? F.at(src, q) : T(0);
                            if (!X.meet()) { gave_up = true; break; }
                        }
                        if (rp >= k) {
                            if (p == k) a[0] = v;
                            else a[1] = v;
                        }
                        if (rp == p) rp = q;
                        else if (rp == q) rp = p;
                        const int m = __shfl_sync(0xffffffffu, from, p - k0);
                        if (orig >= 0) F.at(orig, q) = F.at(orig, k0 + m);
                        if (C > 1) __threadfence();      // (pp_bring reads past the first-level cache)
                    }
                    X.open(X.join_bytes() + (r2 >= 0 ? 2 : 1) * X.row_bytes(left));
                    X.join();
                    X.row(a, spare ? -1 : rp, k, j, left);
                    if (r2 >= 0) X.row(a, spare ? -1 : rp, k + 1, j + 1, left);
                    if (!X.close()) { gave_up = true; break; }
                }
            }
            if (GEN || r2 < 0) {
                double dk = (double)S.prow[j][1];
                int kk = KIND_1X1;
                if (!(fabs(dk) >= pv.eps) || dk == 0.0) {
                    const bool zero = dk == 0.0;
                    int lpk = 0;
                    if (!GEN) {   // the column this row is of
                        X.open(X.join_bytes() + 4);
                        X.join();
                        if (rp == k && !spare)
#pragma unroll 1
                            for (int q = 0; q < C; ++q) X.put(&S.plp, q, mylp);
                        if (!X.close()) { gave_up = true; break; }
                        lpk = S.plp;
                    }
                    const int req = !GEN && pv.psign ? (int)pv.psign[pv.perm[F.c0 + lpk]] : 0;
                    dk = perturb_sign_of(dk, req) * pv.eps;
                    kk = KIND_PERTURBED;
                    if (tid == 0) {
                        S.st[ST_NZERO] += zero;
                        S.st[ST_NPERT]++;
                        if (dk == 0.0 && S.st[ST_INFO] == 0) S.st[ST_INFO] = (GEN ? k : lpk) + 1;
                    }
                }
                if (tid == 0) {
                    S.kind[j] = kk;
                    S.tdk[j] = dk;
                    S.tee[j] = 0.0;
                }
                if (rp > k) {
                    const T l = GEN ? a[0] / T(dk) : T((double)a[0] / dk);
                    S.L[j][tid] = l;
                    const T* row = S.prow[j] + 1;
                    // columns at and beyond `left` hold nothing any more, whatever lands in them
#pragma unroll
                    for (int g = 0; g < PP_NB; g += 16)
                        if (g + 1 < left) {
                            T u[16];   // every load before the first update
#pragma unroll
                            for (int e = 0; e < 16; e += 2)
                                if (g + e + 2 < PP_NB) pp_load2(row + g + e + 1, u[e], u[e + 1]);
                                else u[e] = row[g + e + 1];
#pragma unroll
                            for (int e = 0; e < 16; ++e)
                                if (g + e + 1 < PP_NB) a[g + e] = a[g + e + 1] - l * u[e];
                        }
                }
                j += 1;
            } else {
                if (lane == j) from |= FIRST;
                const double fa = (double)S.prow[j][1], fb = (double)S.prow[j + 1][1], fc = (double)S.prow[j + 1][2];
                const double det = fa * fc - fb * fb;
                const double e11 = fc / det, e12 = -fb / det, e21 = -fb / det, e22 = fa / det;
                if (tid == 0) {
                    S.st[ST_N2X2]++;
                    if (det < 0) { S.st[ST_NPOS]++; S.st[ST_NNEG]++; }
                    else S.st[fa > 0 ? ST_NPOS : ST_NNEG] += 2;
                    S.kind[j] = KIND_2X2_FIRST;
                    S.kind[j + 1] = KIND_2X2_SECOND;
                    S.tdk[j] = fa;
                    S.tdk[j + 1] = fc;
                    S.tee[j] = fb;
                    S.tee[j + 1] = 0.0;
                }
                if (rp == k + 1) S.L[j][tid] = T(0);
                if (rp > k + 1) {
                    const double x1 = (double)a[0], x2 = (double)a[1];
                    const T l1 = T(x1 * e11 + x2 * e21), l2 = T(x1 * e12 + x2 * e22);
                    S.L[j][tid] = l1;
                    S.L[j + 1][tid] = l2;
#pragma unroll
                    for (int e = 0; e < PP_NB - 2; ++e)
                        if (e + 2 < left) a[e] = a[e + 2] - (l1 * S.prow[j][e + 3] + l2 * S.prow[j + 1][e + 3]);
                }
                j += 2;
            }
        }
        if (gave_up && lane == 0) S.fail = 1;
        if (tid == 0) {
            S.nbd = j;
            S.xn = X.xn;
        }
    }
    __syncthreads();
    if (S.fail) return -1;
    if (tid == 0) S.gate = 0;   // for the next block: its group's meetings come first
    F.xn = S.xn;
    const int nbd = S.nbd, k1 = k0 + nbd;
    // the multipliers and what is left of the columns out to the rows' places
    if (orig >= 0 && rp >= k1) {
        for (int e = 0; e < nbd; ++e) F.P[rp + (int64_t)(k0 + e) * f] = S.L[e][tid];
#pragma unroll
        for (int e = 0; e < PP_NB; ++e)
            if (nbd + e < nb) F.P[rp + (int64_t)(k1 + e) * f] = a[e];
        if (rp != orig) {
            const int d = atomicAdd(&F.hdr->ndisp[F.par], 1);
            F.hdr->ddst[d] = rp;
            F.hdr->dsrc[d] = orig;
        }
    } else if (orig >= 0) {
        const int t = rp - k0;
        F.hdr->rowmap[t] = orig;
        for (int s = 0; s < t; ++s) {
            const T l = S.L[s][tid];
            F.P[rp + (int64_t)(k0 + s) * f] = l;
            F.hdr->lt[s][t] = l;
        }
    }
    if (orig >= 0 && rp != orig) F.hdr->moved[F.par] = 1;
    if (orig >= 0 && rp < w) F.lp[rp] = mylp;
    if (rank == 0) {
        if (GEN)
            for (int q = tid; q < nbd * nb; q += PP_THREADS) {
                const int t = q / nb, s = q % nb;        // row t, column s
                if (s > t) F.U[(k0 + s) + (int64_t)(k0 + t) * f] = S.prow[t][1 + s - t] / T(S.tdk[t]);
            }
        if (tid < nbd) {
            F.hdr->kind[tid] = S.kind[tid];
            F.hdr->tdk[tid] = T(S.tdk[tid]);
            F.dd[k0 + tid] = S.tdk[tid];
            if (!GEN) F.ee[k0 + tid] = S.tee[tid];
            F.kd[k0 + tid] = (signed char)S.kind[tid];
        }
        const int kt = tid < nbd ? S.kind[tid] : 0;
        const double dt = tid < nbd && (kt == KIND_1X1 || kt == KIND_PERTURBED) ? S.tdk[tid] : 0.0;
        const unsigned pos = __ballot_sync(0xffffffffu, dt > 0), neg = __ballot_sync(0xffffffffu, dt < 0),
                       two = __ballot_sync(0xffffffffu, kt == KIND_2X2_FIRST);
        if (tid == 0) {
            if (!GEN) {
                S.st[ST_NPOS] += __popc(pos);
                S.st[ST_NNEG] += __popc(neg);
            }
            F.hdr->pairs = two != 0;
            F.hdr->k0 = k0;
            F.hdr->k1 = k1;
            F.hdr->kend = kend;
        }
    }
    return k1;
}

// T1: the block's rows right of the block, solved against its unit triangle (unscaled, into F.us); the rows'
// interchanges in the columns left of the block
template <typename T, int STRUCT>
__device__ void pp_rows(const PanelFront<T, STRUCT == STRUCT_G>& F, const PanelHdr<T>& H) {
    constexpr bool GEN = STRUCT == STRUCT_G;
    const int f = F.f, nbd = H.k1 - H.k0;
    const int lane = threadIdx.x & 31, gt = F.grank * PP_THREADS + threadIdx.x, GT = F.gs * PP_THREADS;
    const int cfirst = GEN ? H.k1 : H.kend, clast = GEN ? f : F.w;
    // Four lanes per column, row 4 i + sub in a lane's g[i]: the solve is a chain of nbd broadcasts, 1 us for a
    // warp, where one lane per column took 3; eight columns a warp, the warps spread over the group's CTAs
    // (sixteen in one CTA took 16 us).
    constexpr int NG = PP_NB / 4;
    const int sub = lane & 3;
    for (int c0 = cfirst + ((threadIdx.x >> 5) * F.gs + F.grank) * 8; c0 < clast; c0 += F.gs * PP_WARPS * 8) {
        const int c = c0 + (lane >> 2);
        const bool live = c < clast;
        T g[NG];
#pragma unroll
        for (int i = 0; i < NG; ++i) {
            const int t = 4 * i + sub;
            g[i] = live && t < nbd ? F.at(H.moved[F.par] ? H.rowmap[t] : H.k0 + t, c) : T(0);
        }
        if (!H.pairs) {
            for (int s = 0; s < nbd; s += 4) {
                T l[4][NG];   // every multiplier of the four columns before the chain
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int i = 0; i < NG; ++i) l[q][i] = s + 4 * i < PP_NB ? H.lt[s + q][s + sub + 4 * i] : T(0);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const T u = __shfl_sync(0xffffffffu, g[0], (lane & ~3) + q);
                    if (live && sub == q && s + q < nbd) F.us[(int64_t)(s + q) * f + c] = u;
#pragma unroll
                    for (int i = 0; i < NG; ++i)
                        if (i > 0 || sub > q) g[i] -= l[q][i] * u;   // rows beyond nbd are never used
                }
#pragma unroll
                for (int i = 0; i + 1 < NG; ++i) g[i] = g[i + 1];
            }
            continue;
        }
        T u0 = T(0);   // the first of a 2x2 pair's two rows
        for (int s = 0; s < nbd; s += 4) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (s + q >= nbd) break;
                const T u = __shfl_sync(0xffffffffu, g[0], (lane & ~3) + q);
                if (live && sub == q) F.us[(int64_t)(s + q) * f + c] = u;
                const T* l = &H.lt[s + q][s + sub];
                const int kd = H.kind[s + q];
                if (kd == KIND_2X2_FIRST) {
                    u0 = u;
                } else if (kd == KIND_2X2_SECOND) {
                    const T* l0 = &H.lt[s + q - 1][s + sub];
#pragma unroll
                    for (int i = 0; i < NG; ++i)
                        if (s + 4 * i < nbd && (i > 0 || sub > q)) g[i] -= l0[4 * i] * u0 + l[4 * i] * u;
                } else {
#pragma unroll
                    for (int i = 0; i < NG; ++i)
                        if (s + 4 * i < nbd && (i > 0 || sub > q)) g[i] -= l[4 * i] * u;
                }
            }
#pragma unroll
            for (int i = 0; i + 1 < NG; ++i) g[i] = g[i + 1];
        }
    }
    if (!H.moved[F.par]) return;
    for (int c = gt; c < H.k0; c += GT) {
        T* col = F.P + (int64_t)c * f;
        T b[2 * PP_NB];
        for (int t = 0; t < nbd; ++t) b[t] = col[H.rowmap[t]];
        for (int d = 0; d < H.ndisp[F.par]; ++d) b[PP_NB + d] = col[H.dsrc[d]];
        for (int t = 0; t < nbd; ++t) col[H.k0 + t] = b[t];
        for (int d = 0; d < H.ndisp[F.par]; ++d) col[H.ddst[d]] = b[PP_NB + d];
    }
}

// One update tile: entries (row0 + i, col0 + c) of `C` (leading dimension f), each minus the block's
// products R[row] Cc[col] in the order of its columns. R and Cc are read at R[row + t rld] and
// Cc[col + t cld]. Entry (row, col) is live when row >= col + low. src(row, col): where its value comes from.
template <typename T, int STRUCT, int RI, class SRC>
__device__ __forceinline__ void pp_tile(PanelSmem<T>& S, const PanelHdr<T>& H, T* Cp, int f, int row0, int col0, int nr,
                                        int nc, int low, const T* R, int64_t rld, const T* Cc, int64_t cld, SRC src) {
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5, nbd = H.k1 - H.k0;
    T c[RI][4];
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = tx + 32 * i, cc = 4 * ty + q;
            c[i][q] = r < nr && cc < nc && row0 + r >= col0 + cc + low ? *src(row0 + r, col0 + cc) : T(0);
        }
    constexpr int TR = 32 * RI;
#pragma unroll
    for (int x = 0; x < PP_NB * TR / PP_THREADS; ++x) {
        const int q = tid + x * PP_THREADS, t = q / TR, r = q % TR;
        S.Rs[t][r] = t < nbd && r < nr ? R[row0 + r + (int64_t)t * rld] : T(0);
    }
#pragma unroll
    for (int x = 0; x < PP_NB * PP_TC / PP_THREADS; ++x) {
        const int q = tid + x * PP_THREADS, t = q / PP_TC, r = q % PP_TC;
        S.Cs[t][r] = t < nbd && r < nc ? Cc[col0 + r + (int64_t)t * cld] : T(0);
    }
    __syncthreads();
    if (STRUCT != STRUCT_S || !H.pairs) {
#pragma unroll 4
        for (int t = 0; t < PP_NB; ++t) {   // beyond nbd: zeros
            T ra[RI], ca[4];
#pragma unroll
            for (int i = 0; i < RI; ++i) ra[i] = S.Rs[t][tx + 32 * i];
#pragma unroll
            for (int q = 0; q < 4; ++q) ca[q] = S.Cs[t][4 * ty + q];
#pragma unroll
            for (int i = 0; i < RI; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) c[i][q] -= ra[i] * ca[q];
        }
    }
    for (int t = STRUCT != STRUCT_S || !H.pairs ? nbd : 0; t < nbd;) {
        T ra[RI], ca[4];
#pragma unroll
        for (int i = 0; i < RI; ++i) ra[i] = S.Rs[t][tx + 32 * i];
#pragma unroll
        for (int q = 0; q < 4; ++q) ca[q] = S.Cs[t][4 * ty + q];
        if (STRUCT == STRUCT_S && H.kind[t] == KIND_2X2_FIRST) {
            T rb[RI], cb[4];
#pragma unroll
            for (int i = 0; i < RI; ++i) rb[i] = S.Rs[t + 1][tx + 32 * i];
#pragma unroll
            for (int q = 0; q < 4; ++q) cb[q] = S.Cs[t + 1][4 * ty + q];
#pragma unroll
            for (int i = 0; i < RI; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) c[i][q] -= ra[i] * ca[q] + rb[i] * cb[q];
            t += 2;
        } else {
#pragma unroll
            for (int i = 0; i < RI; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) c[i][q] -= ra[i] * ca[q];
            t += 1;
        }
    }
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = tx + 32 * i, cc = 4 * ty + q;
            if (r < nr && cc < nc && row0 + r >= col0 + cc + low) Cp[row0 + r + (int64_t)(col0 + cc) * f] = c[i][q];
        }
    __syncthreads();
}

// T2: the block's products into the rest of the front. "S": columns kend .. w - 1, rows k1 .. f - 1. "G": the
// same columns (k1 .. w - 1) on and below the diagonal in the L panel, and rows k1 .. w - 1 right of the
// diagonal in the U^T panel (there a tile's rows are the matrix' columns).
template <typename T, int STRUCT, int RI>
__device__ void pp_update_tiles(const PanelFront<T, STRUCT == STRUCT_G>& F, PanelSmem<T>& S, const PanelHdr<T>& H) {
    constexpr bool GEN = STRUCT == STRUCT_G;
    const int f = F.f, w = F.w, k1 = H.k1, cf = GEN ? k1 : H.kend;
    constexpr int TR = 32 * RI;
    const int ntr = (f - k1 + TR - 1) / TR, ntc = (w - cf + PP_TC - 1) / PP_TC;
    const int nt = ntr * ntc, all = GEN ? 2 * nt : nt;
    const T* Lb = F.P + (int64_t)H.k0 * f;
    const int ndisp = H.ndisp[F.par];
    auto row_of = [&](int i) {
        int s = i;
        for (int d = 0; d < ndisp; ++d)
            if (H.ddst[d] == i) s = H.dsrc[d];
        return s;
    };
    for (int q = F.grank; q < all; q += F.gs) {
        const int qq = q < nt ? q : q - nt;
        const int row0 = k1 + (qq % ntr) * TR, col0 = cf + (qq / ntr) * PP_TC;
        const int nr = min(TR, f - row0), nc = min(PP_TC, w - col0);
        if (GEN && row0 + nr - 1 < col0) continue;   // above the diagonal
        if (q < nt) {
            pp_tile<T, STRUCT, RI>(S, H, F.P, f, row0, col0, nr, nc, GEN ? 0 : -(1 << 29), Lb, f, F.us, f,
                               [&](int i, int c) -> const T* {
                                   const int s = row_of(i);
                                   return s == i ? F.P + i + (int64_t)c * f : &F.at(s, c);
                               });
        } else if constexpr (GEN) {
            pp_tile<T, STRUCT, RI>(S, H, F.U, f, row0, col0, nr, nc, 1, F.us, f, Lb, f,
                               [&](int c, int i) -> const T* { return F.U + c + (int64_t)row_of(i) * f; });
        }
    }
}

template <typename T, int STRUCT>
__device__ void pp_update(const PanelFront<T, STRUCT == STRUCT_G>& F, PanelSmem<T>& S, const PanelHdr<T>& H) {
    const int cf = STRUCT == STRUCT_G ? H.k1 : H.kend;
    if (cf >= F.w) return;
    // 128-row tiles (fewer operand bytes per entry) unless 64-row tiles end in fewer half rounds
    const int sides = STRUCT == STRUCT_G ? 2 : 1, ntc = (F.w - cf + PP_TC - 1) / PP_TC, m = F.f - H.k1;
    const int n4 = sides * ((m + PP_TR - 1) / PP_TR) * ntc, n2 = sides * ((m + PP_TR / 2 - 1) / (PP_TR / 2)) * ntc;
    if (2 * ((n4 + F.gs - 1) / F.gs) <= (n2 + F.gs - 1) / F.gs) pp_update_tiles<T, STRUCT, 4>(F, S, H);
    else pp_update_tiles<T, STRUCT, 2>(F, S, H);
}

// "G": the block's rows, scaled, into the U^T panel (after T2: its tiles may read the rows' old values)
template <typename T>
__device__ void pp_urows(const PanelFront<T, true>& F, const PanelHdr<T>& H, int part, int nparts) {
    const int nbd = H.k1 - H.k0, n = F.f - H.k1;
    const int64_t gt = (int64_t)part * PP_THREADS + threadIdx.x, GT = (int64_t)nparts * PP_THREADS;
    for (int64_t q = gt; q < (int64_t)n * nbd; q += GT) {
        const int t = (int)(q / n), c = H.k1 + (int)(q % n);
        F.U[c + (int64_t)(H.k0 + t) * F.f] = F.us[(int64_t)t * F.f + c] / H.tdk[t];
    }
}

// One front, by every CTA of its group
template <typename T, int STRUCT>
__device__ void pp_front(const LargePivotArgs<T>& A, const PanelJob& job, PanelSmem<T>& S, const PanelGroups& G,
                         unsigned& xn) {
    constexpr bool GEN = STRUCT == STRUCT_G;
    const int C = G.csize;
    const int s = A.list[job.fi];
    const DFront fd = A.fronts[s];
    PanelFront<T, GEN> F;
    const int f = fd.f, w = fd.w, ncta = job.role == PANEL_SINGLE ? 1 : C;
    F.P = A.factor + fd.panel;
    F.U = GEN ? A.ufactor + fd.panel : nullptr;
    F.f = f;
    F.w = w;
    F.c0 = fd.c0;
    double* scr = A.scratch + A.scr_off[job.fi];
    F.dd = scr;
    F.ee = scr + w;
    F.lp = reinterpret_cast<int*>(F.ee + w);
    F.kd = reinterpret_cast<signed char*>(F.ee + w + (w + 1) / 2);
    double* h = F.ee + w + (w + 1) / 2 + (w + 7) / 8;
    F.hdr = reinterpret_cast<PanelHdr<T>*>(h);
    F.us = reinterpret_cast<T*>(h + sizeof(PanelHdr<double>) / 8 + 1);
    F.C = ncta;
    F.rank = job.rank < ncta ? job.rank : 0;
    F.gs = job.gs;
    F.grank = job.rank;
    F.xn = xn;
    F.par = 0;
    F.bar = G.bar + job.fi;
    F.epoch = &S.epoch;
    F.limit = &S.limit;
    F.ok = &S.ok;
    F.dead = &S.dead;
    if (threadIdx.x == 0) {
        S.ok = 1;
        S.limit = {G.status, G.wait_ns};
        S.gate = S.fail = 0;
        S.epoch = 0;
        for (int q = 0; q < NSTAT; ++q) S.st[q] = 0;
    }
    __syncthreads();
    const bool leads = job.rank < ncta;
    const int tid = threadIdx.x, gt = job.rank * PP_THREADS + tid, GT = job.gs * PP_THREADS;
    const PanelPivot pv{A.pivot, A.lu_pivot, A.u, A.eps, A.psign, A.perm};
    if (STRUCT == STRUCT_S)
        for (int64_t q = gt; q < (int64_t)w * w; q += GT) {
            const int i = (int)(q % w), j = (int)(q / w);
            if (i > j) F.P[j + (int64_t)i * f] = F.P[i + (int64_t)j * f];
        }
    for (int q = gt; q < w; q += GT) F.lp[q] = q;
    if (gt == 0) F.hdr->ndisp[0] = F.hdr->moved[0] = 0;
    PanelHdr<T>& H = S.hdr;
    // A wait that gave up (a status word, no fault) ends the front. With helper clusters, whose meetings are in
    // global memory, each CTA leaves by itself: the cluster's next barrier is the kernel's, behind the front.
    // Without, the meetings are cluster barriers, and its CTAs leave together, at the one behind the exchanges:
    // nobody can set `dead` between that barrier and its look at it.
    const bool alone = F.gs == F.C;
    bool ok = pp_group_sync(F);
    for (int k = 0, first = 1; ok && k < w; first = 0, F.par ^= 1) {
        if constexpr (GEN) {   // the previous block's rows: the helpers while the leader factors, or everyone
            const int helpers = F.gs - F.C;
            if (!first && helpers == 0) pp_urows<T>(F, H, F.grank, F.gs);
            else if (!first && !leads) pp_urows<T>(F, H, F.grank - F.C, helpers);
        }
        int k1 = 0;
        if (leads) k1 = pp_block<T, STRUCT>(F, S, pv, k);
        if (k1 < 0) pp_give_up(F);
        ok = alone || k1 >= 0;
        if (ok) ok = pp_group_sync(F);
        if (alone) ok = *(volatile int*)F.dead == 0;
        if (!ok) break;
        const int* src = reinterpret_cast<const int*>(F.hdr);
        int* dst = reinterpret_cast<int*>(&H);
        for (int q = tid; q < (int)(sizeof(PanelHdr<T>) / 4); q += PP_THREADS) dst[q] = src[q];
        __syncthreads();
        k = H.k1;
        pp_rows<T, STRUCT>(F, H);
        ok = pp_group_sync(F);
        if (ok && k < w) {
            pp_update<T, STRUCT>(F, S, H);
            ok = pp_group_sync(F);
        }
    }
    if (!ok) {
        pp_give_up(F);
        return;
    }
    if (F.C > 1) xn = F.xn;   // one CTA alone uses no mbarrier
    if constexpr (GEN) pp_urows<T>(F, H, F.grank, F.gs);
    for (int64_t q = gt; q < (int64_t)w * w; q += GT) {
        const int i = (int)(q % w), j = (int)(q / w);
        if (i == j) {
            F.P[i + (int64_t)j * f] = T(1);
            if (GEN) F.U[i + (int64_t)j * f] = T(1);
        } else if (i < j && !GEN) {
            F.P[i + (int64_t)j * f] = T(0);
        }
    }
    const int64_t n = A.n;
    for (int q = gt; q < w; q += GT) {
        const int64_t g = fd.c0 + q;
        A.piv[g] = fd.c0 + F.lp[q] + 1;
        A.kind[g] = F.kd[q];
        A.d[g] = F.dd[q];
        A.d[n + g] = STRUCT == STRUCT_S ? F.ee[q] : 0.0;
    }
    if (F.grank == 0 && tid == 0) {
        int64_t* So = A.stats + (int64_t)s * NSTAT;
        for (int q = 0; q < NSTAT; ++q) So[q] = S.st[q];
        A.finfo[s] = S.st[ST_INFO];
    }
}

}  // namespace sds
