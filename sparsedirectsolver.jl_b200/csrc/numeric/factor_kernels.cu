// Fused per-front kernels of the numeric phase.
//
// small_front_kernel: one CTA per front of one level, the whole f x f front in
// shared memory: zero, assemble A, extend-add the children's contribution
// blocks (children in child_list order, so every sum has a fixed order and the
// result is bitwise reproducible), the dense partial factorization of the w
// fully-summed columns (Cholesky; Bunch-Kaufman LDLT; threshold-pivoting LU),
// the Schur update of the contribution block, and the write-out of the panel,
// D, pivots, statistics and contribution block. It replaces the reference's
// regime B kernels (front_cholesky_kernel! src/numeric/front.jl:154-206,
// front_ldlt_kernel! src/numeric/ldlt.jl:992-1111, front_lu_kernel!
// src/numeric/lu.jl:264-330); the in-front arithmetic follows the CPU reference
// (src/reference/*.jl) step by step.
//
// subtree_kernel: the same per-front body run by one CTA over a whole leaf
// subtree of such fronts in postorder (the reference's regime A).
//
// warp_front_kernel: Cholesky fronts of at most 32 rows, one warp per front, for
// level launches of many such fronts (batches of small systems).
//
// assemble_large_kernel: column-owner assembly of the fronts too large for
// shared memory: one warp per (front, parent index p) builds the column it
// owns in row chunks from the entries of A of that column and every child's
// contribution, in child order. No atomics.
#include <cuda_runtime.h>
#include <math.h>
#include <math_constants.h>
#include <stdint.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "front_factor.cuh"
#include "pivot.cuh"

namespace sds {

// The pivot of a Cholesky column: d = max(ajj, eps), its reciprocal square root and square root. False: it fails.
__device__ __forceinline__ bool spd_pivot(double ajj, double eps, double& r, double& root) {
    const bool ok = ajj > eps || (eps > 0 && ajj >= 0);
    const double d = fmax(ajj, eps);
    r = fast_rsqrt(d);
    if (!fast_rsqrt_ok(d)) r = rsqrt(d);
    root = d * r;   // and Newton's correction, off the chain of columns
    root = d < CUDART_INF ? fma(fma(-root, root, d), 0.5 * r, root) : d;
    return ok;
}

// The in-front Cholesky of a front of at most 32 RPL rows by eight warps, in registers: warp q holds the
// columns p = q (mod 8), lane the rows lane + 32 i. Per column one exchange: the owner scales it by the
// reciprocal square root and puts it in shared memory (two buffers, one barrier); every warp updates its
// later columns, the owner of the next one that column first, so that its pivot is on its way meanwhile.
// What bounds it: that chain while few fronts are in flight, the FP64 units with many: 768 fronts of 96 rows
// 63 us (the columns as a loop that the compiler did not unroll, the registers in local memory: 253 us; one front
// by itself 0.35 us a column in shared memory with three barriers, 0.2 in registers). Returns 0, or 1 + the
// column whose pivot fails.
template <typename T, int RPL>
struct SpdRegs {
    static constexpr int CPW = 4 * RPL, R = 32 * RPL;
    T (&a)[CPW][RPL];
    const int w, lane, warp;
    const double eps;
    T* const lcol;
    volatile int* const fail;

    // this warp's column k in a[c]: final, and into its buffer
    template <int c>
    __device__ __forceinline__ void scale(int k) {
        constexpr int i0 = (8 * c) >> 5;   // the row chunk of row k
        double r, root;
        if (!spd_pivot((double)__shfl_sync(0xffffffffu, a[c][i0], k & 31), eps, r, root)) {
            if (lane == 0) fail[k & 1] = k + 1;   // read after the next barrier; the other word until then
            return;
        }
        T* l = lcol + (k & 1) * R;
#pragma unroll
        for (int i = 0; i < RPL; ++i) {
            a[c][i] *= T(r);   // rows above k are never read
            l[lane + 32 * i] = a[c][i];
        }
        if (lane == (k & 31)) a[c][i0] = T(root);
    }
    template <int c>
    __device__ __forceinline__ void update(const T* l, const T (&li)[RPL], int p) {
        const T lp = l[p];
#pragma unroll
        for (int i = 0; i < RPL; ++i) a[c][i] = fma(-li[i], lp, a[c][i]);
    }
    template <int c, int c1>
    __device__ __forceinline__ void update_from(const T* l, const T (&li)[RPL]) {
        if constexpr (c < c1) {
            update<c>(l, li, 8 * c + warp);
            update_from<c + 1, c1>(l, li);
        }
    }
    // the columns n = 8 c .. : the update by column n - 1, the next pivot first (as a recursion over c: every
    // register index is a constant)
    template <int c>
    __device__ __forceinline__ int columns() {
        if constexpr (c < CPW) {
            for (int q = 0; q < 8; ++q) {
                const int n = 8 * c + q, k = n - 1;
                if (n > w) return 0;
                const T* l = lcol + (k & 1) * R;
                T li[RPL];
                if (c > 0 || q > 0) {
                    __syncthreads();
                    if (const int at = fail[k & 1]) return at;
#pragma unroll
                    for (int i = 0; i < RPL; ++i) li[i] = l[lane + 32 * i];
                    if (warp >= q) update<c>(l, li, 8 * c + warp);
                }
                if (warp == q && n < w) scale<c>(n);
                if (c > 0 || q > 0) update_from<c + 1, CPW>(l, li);
            }
            return columns<c + 1>();
        }
        // a front that fills the registers: its last column's pivot
        __syncthreads();
        return w == 8 * CPW ? fail[(w - 1) & 1] : 0;
    }
};

template <typename T, int RPL>
__device__ __forceinline__ int spd_front_regs(T (&a)[4 * RPL][RPL], int w, double eps, T* lcol, volatile int* fail) {
    SpdRegs<T, RPL> f{a, w, (int)threadIdx.x & 31, (int)threadIdx.x >> 5, eps, lcol, fail};
    return f.template columns<0>();
}

// One front by the whole CTA, in shared memory (smem_raw holds at least small_front_smem(f)). The CTA's
// threads all call it; it ends with the front's outputs written to global memory. RPL > 0: a Cholesky front
// of at most 32 RPL rows, factored in registers by 256 threads.
//
// The bottom levels are launches of a few dependent loads per front, so the loads that do not depend on one
// another go out together: the record; then the kids, rows, items and entries of A; then every contribution.
// (Children one after another, each behind its descriptor, its rows and a barrier: lap2d 16^2 218 us a
// factorization, now 140; lap2d 64^2 1048, now 612; 256 uneven FP32 systems 2530, now 1680. Three launches in
// four are still latency: 5 us each.)
template <typename T, int STRUCT, int RPL>
__device__ __forceinline__ void small_front(const SmallArgs<T>& A, const int at, const int member,
                                            unsigned char* smem_raw) {
    const SFront fd = A.sf[at];
    const int s = fd.s;
    const int f = fd.f, w = fd.w, m = f - w;
    const int ld = f | 1;
    T* F = reinterpret_cast<T*>(smem_raw);
    size_t off = ((size_t)ld * f * sizeof(T) + 15) & ~size_t(15);
    const int max_kids = sf_kids(A.fmax), max_items = sf_items(A.fmax);
    SKid* skid = reinterpret_cast<SKid*>(smem_raw + off);
    uint32_t* sitem = reinterpret_cast<uint32_t*>(skid + max_kids);
    uint8_t* ssri = reinterpret_cast<uint8_t*>(sitem + max_items);
    double* dd = reinterpret_cast<double*>(ssri + max_items); // w
    double* ee = dd + w;                                     // w
    double* lvec = ee + w;                                   // 2 f (multipliers)
    int* lp = reinterpret_cast<int*>(lvec + 2 * f);          // w
    // control words; with the front in registers behind the two column buffers (at dd)
    int* ctl = RPL > 0 ? reinterpret_cast<int*>(reinterpret_cast<T*>(dd) + 64 * RPL) : lp + f;
    signed char* kd = reinterpret_cast<signed char*>(ctl + 16);

    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nt >> 5;
    const double* nz = A.nzval + (int64_t)member * A.nnz;
    T* factor = A.factor + (int64_t)member * A.factor_len;
    T* cbar = A.cb + (int64_t)member * A.cb_len;

    // this thread's first entry of A, on its way while the front is cleared
    int k = fd.am_begin + tid, code = 0, before = 0;
    double v0 = 0.0;
    if (k < fd.am_end) {
        code = A.maps.am_loc[k];
        before = k > fd.am_begin ? A.maps.am_loc[k - 1] : 0;
        v0 = nz[A.maps.am_src[k]];
    }
    const bool skids = fd.nkid <= max_kids, sits = fd.nsri <= max_items;
    if (skids && tid < fd.nkid) skid[tid] = A.kids[fd.kid_begin + tid];
    if (sits)
        for (int q = tid; q < fd.nsri; q += nt) {
            sitem[q] = A.items[fd.sri_begin + q];
            ssri[q] = A.sri[fd.sri_begin + q];
        }
    const SKid* kids = skids ? skid : A.kids + fd.kid_begin;
    const uint32_t* items = sits ? sitem : A.items + fd.sri_begin;
    const uint8_t* sri = sits ? ssri : A.sri + fd.sri_begin;
    for (int q = tid; q < ld * f; q += nt) F[q] = T(0);
    if (tid < 16) ctl[tid] = 0;
    __syncthreads();
    // assembly of A: each run of equal destinations is summed by one thread, in entry order
    for (; k < fd.am_end; k += nt) {
        if (k != fd.am_begin + tid) {
            code = A.maps.am_loc[k];
            before = A.maps.am_loc[k - 1];
            v0 = nz[A.maps.am_src[k]];
        }
        if (before == code) continue;
        T acc = T(0);
        acc += T(v0);
        for (int q = k + 1; q < fd.am_end && A.maps.am_loc[q] == code; ++q) acc += T(nz[A.maps.am_src[q]]);
        int loc = (code > 0 ? code : -code) - 1;
        int i = loc % f, j = loc / f;
        if (code > 0) F[i + j * ld] += acc;
        else F[j + i * ld] += acc;
    }
    // extend-add: a warp's columns, item after item, the first 64 rows of SF_U items loaded before the first
    // addition (and the first of all before the barrier behind the entries of A)
    constexpr int SF_U = 4;
    T v[SF_U][2];
    int n[SF_U], q0[SF_U], p[SF_U];
    const T* col[SF_U];
    const uint8_t* ri[SF_U];
    // (four warps have the items of two groups of columns each; fronts in registers have eight)
    const bool two = RPL == 0 && nwarps < 8;
    const int32_t* ep = A.ep + fd.ep_begin + warp;
    const int e0 = ep[0], n0 = ep[1] - e0, e1 = two ? ep[4] : 0, nitems = n0 + (two ? ep[5] - e1 : 0);
    int e = 0;
    auto load = [&]() {
#pragma unroll
        for (int u = 0; u < SF_U; ++u) {
            n[u] = 0;
            if (e + u >= nitems) continue;
            const uint32_t it = items[!two || e + u < n0 ? e0 + e + u : e1 + e + u - n0];
            const SKid kid = kids[(it >> 8) & 0xffffu];
            const int t = it & 0xffu;
            p[u] = it >> 24;
            q0[u] = STRUCT == STRUCT_G ? 0 : t;
            n[u] = kid.mc;
            col[u] = cbar + kid.cb + (int64_t)t * kid.mc;
            ri[u] = sri + kid.sri;
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int q = q0[u] + lane + 32 * x;
                v[u][x] = q < n[u] ? col[u][q] : T(0);
            }
        }
    };
    if (fd.nsri > 0) load();
    __syncthreads();
    while (fd.nsri > 0) {
#pragma unroll
        for (int u = 0; u < SF_U; ++u) {
            if (n[u] == 0) continue;
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int q = q0[u] + lane + 32 * x;
                if (q < n[u]) F[ri[u][q] + p[u] * ld] += v[u][x];
            }
            constexpr int SF_T = RPL > 0 ? 1 : 4;   // (fronts in registers have at most 96 rows)
            for (int q = q0[u] + lane + 64; q < n[u]; q += 32 * SF_T) {
                T t[SF_T];
#pragma unroll
                for (int x = 0; x < SF_T; ++x) t[x] = q + 32 * x < n[u] ? col[u][q + 32 * x] : T(0);
#pragma unroll
                for (int x = 0; x < SF_T; ++x)
                    if (q + 32 * x < n[u]) F[ri[u][q + 32 * x] + p[u] * ld] += t[x];
            }
            __syncwarp();
        }
        e += SF_U;
        if (e >= nitems) break;
        load();
    }
    if (fd.nsri > 0) __syncthreads();   // (not for the leaves)
    if constexpr (RPL > 0) {
        constexpr int CPW = 4 * RPL;
        T a[CPW][RPL];
#pragma unroll
        for (int c = 0; c < CPW; ++c)
#pragma unroll
            for (int i = 0; i < RPL; ++i) {
                const int p = 8 * c + warp, r = lane + 32 * i;
                a[c][i] = (p < f && r < f && r >= p) ? F[r + p * ld] : T(0);
            }
        const int status = spd_front_regs<T, RPL>(a, w, A.eps, reinterpret_cast<T*>(dd), ctl);
        T* P = factor + fd.panel;
        const bool cbw = fd.cb >= 0 && m > 0 && status == 0;
        T* C = cbar + fd.cb;
#pragma unroll
        for (int c = 0; c < CPW; ++c)
#pragma unroll
            for (int i = 0; i < RPL; ++i) {
                const int p = 8 * c + warp, r = lane + 32 * i;
                if (p < w) {
                    if (r < f) P[r + (int64_t)p * f] = r < p ? T(0) : a[c][i];
                } else if (cbw && p < f && r < f && r >= p) {
                    C[(r - w) + (int64_t)(p - w) * m] = a[c][i];
                }
            }
        if (tid == 0) {
            int64_t* S = A.stats + ((int64_t)member * A.ns + s) * NSTAT;
            for (int q = 0; q < NSTAT; ++q) S[q] = q == ST_NPOS ? (status ? status - 1 : w) : q == ST_INFO ? status : 0;
            A.finfo[(int64_t)member * A.ns + s] = status;
        }
        return;
    }
    if (STRUCT == STRUCT_S) {  // the pivoting reads both triangles of the fully-summed block
        for (int q = tid; q < w * w; q += nt) {
            int i = q % w, j = q / w;
            if (i > j) F[j + i * ld] = F[i + j * ld];
        }
        __syncthreads();
    }
    int64_t st[NSTAT] = {0, 0, 0, 0, 0, 0};
    int status = 0;
    const double eps = A.eps;

    if (STRUCT == STRUCT_SPD) {
        for (int j = 0; j < w; ++j) {
            double ajj = (double)F[j + j * ld];
            bool ok = ajj > eps || (eps > 0 && ajj >= 0);
            if (!ok) { status = j + 1; break; }
            double djj = sqrt(fmax(ajj, eps));
            T inv = T(1.0 / djj);
            __syncthreads();
            for (int i = j + 1 + tid; i < f; i += nt) F[i + j * ld] *= inv;
            if (tid == 0) F[j + j * ld] = T(djj);
            __syncthreads();
            for (int l = j + 1 + warp; l < f; l += nwarps) {
                const T flj = F[l + j * ld];
                for (int i = l + lane; i < f; i += 32) F[i + l * ld] -= F[i + j * ld] * flj;
            }
            __syncthreads();
        }
        st[ST_NPOS] = status ? status - 1 : w;
        st[ST_INFO] = status;
    } else if (STRUCT == STRUCT_S) {
        SmemStore<T> store{F, ld, f, w};
        FrontScratch sc{lvec, dd, ee, lp, kd, ctl};
        ldlt_front_steps<T>(store, sc, f, w, A.pivot, A.u, eps, A.psign, A.maps.perm, fd.c0, st);
        // F22 -= (L21 D) L21^T, lower triangle, kk in order (ldlt.jl:184-191)
        for (int jj = warp; jj < m; jj += nwarps)
            for (int ii = jj + lane; ii < m; ii += 32) {
                T acc = F[w + ii + (w + jj) * ld];
                int q = 0;
                while (q < w) {
                    if (kd[q] == KIND_2X2_FIRST) {
                        double x1 = (double)F[w + ii + q * ld], x2 = (double)F[w + ii + (q + 1) * ld];
                        T w1 = T(x1 * dd[q] + x2 * ee[q]), w2 = T(x1 * ee[q] + x2 * dd[q + 1]);
                        acc -= w1 * F[w + jj + q * ld];
                        acc -= w2 * F[w + jj + (q + 1) * ld];
                        q += 2;
                    } else {
                        acc -= T((double)F[w + ii + q * ld] * dd[q]) * F[w + jj + q * ld];
                        q += 1;
                    }
                }
                F[w + ii + (w + jj) * ld] = acc;
            }
        __syncthreads();
    } else {  // STRUCT_G: LU with row interchanges inside the fully-summed rows
        SmemStore<T> store{F, ld, f, w};
        FrontScratch sc{lvec, dd, ee, lp, kd, ctl};
        lu_front_steps<T>(store, sc, f, w, A.lu_pivot != 0, A.u, eps, st);
        // F22 -= (L21 D) U12, summed over k in order (lu.jl:142-150)
        for (int jj = warp; jj < m; jj += nwarps)
            for (int ii = lane; ii < m; ii += 32) {
                T acc = T(0);
                for (int q = 0; q < w; ++q) acc += F[w + ii + q * ld] * T(dd[q]) * F[q + (w + jj) * ld];
                F[w + ii + (w + jj) * ld] -= acc;
            }
        __syncthreads();
    }

    // write-out: panel (and U^T panel), D / pivots, statistics, contribution block
    T* P = factor + fd.panel;
    const bool unit = STRUCT != STRUCT_SPD;
    for (int j = warp; j < w; j += nwarps)
        for (int i = lane; i < f; i += 32) {
            T v = i < j ? T(0) : (i == j && unit ? T(1) : F[i + j * ld]);
            P[i + (int64_t)j * f] = v;
        }
    if (STRUCT == STRUCT_G) {
        T* U = A.ufactor + (int64_t)member * A.factor_len + fd.panel;
        for (int j = warp; j < w; j += nwarps)
            for (int i = lane; i < f; i += 32) U[i + (int64_t)j * f] = i < j ? T(0) : (i == j ? T(1) : F[j + i * ld]);
    }
    if (STRUCT != STRUCT_SPD) {
        const int64_t n = A.n;
        for (int q = tid; q < w; q += nt) {
            const int64_t g = fd.c0 + q;
            A.piv[member * n + g] = fd.c0 + lp[q] + 1;
            A.kind[member * n + g] = kd[q];
            A.d[member * 2 * n + g] = dd[q];
            A.d[member * 2 * n + n + g] = STRUCT == STRUCT_S ? ee[q] : 0.0;
        }
    }
    if (tid == 0) {
        int64_t* S = A.stats + ((int64_t)member * A.ns + s) * NSTAT;
        for (int q = 0; q < NSTAT; ++q) S[q] = st[q];
        A.finfo[(int64_t)member * A.ns + s] = (int32_t)st[ST_INFO];
    }
    if (fd.cb >= 0 && m > 0 && status == 0) {
        T* C = cbar + fd.cb;
        for (int jj = warp; jj < m; jj += nwarps)
            for (int ii = (STRUCT == STRUCT_G ? 0 : jj) + lane; ii < m; ii += 32)
                C[ii + (int64_t)jj * m] = F[w + ii + (w + jj) * ld];
    }
}

// CTAs of 256 threads that an SM must hold: levels and batches of small fronts need them more than the registers
// (lap2d 300^2 a pass 2.02 ms, 2.08 with 82 and 85 registers where 64 and 80 fit; 128 systems of lap2d 48^2 "S" 2.20 ms,
// 2.38 with 80).
constexpr int small_front_ctas(int rpl) { return rpl == 1 ? 3 : rpl == 3 ? 2 : 4; }
template <typename T, int STRUCT, int RPL>
__global__ void __launch_bounds__(256, small_front_ctas(RPL)) small_front_kernel(SmallArgs<T> A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int member = A.members ? A.members[blockIdx.y] : blockIdx.y;
    small_front<T, STRUCT, RPL>(A, blockIdx.x, member, smem_raw);
}

// Fused subtrees: one CTA factors a whole subtree of shared-memory fronts, front after front in the
// subtree's postorder (A.sf[A.sub_ptr[b] .. A.sub_ptr[b + 1]) for CTA b), in one launch for every
// subtree of its size class instead of one launch per level. A child's contribution block goes to
// global memory (the subtree's stack region of the arena, hot in L2) and its parent, later in the same
// CTA, reads it back after the barrier between the two fronts, which makes the CTA's global writes
// visible to all its threads. Each front's arithmetic is small_front's, so the factor is bit for bit
// the level launches'. Replaces the reference's regime-A kernels (subtree_cholesky_kernel!
// src/numeric/subtree.jl:274-316, subtree_ldlt_kernel! src/numeric/ldlt.jl:1133-1228,
// subtree_lu_kernel! src/numeric/lu.jl:424-493).
template <typename T, int STRUCT, int RPL>
__global__ void __launch_bounds__(256, small_front_ctas(RPL)) subtree_kernel(SmallArgs<T> A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int member = A.members ? A.members[blockIdx.y] : blockIdx.y;
    const int q0 = A.sub_ptr[blockIdx.x], q1 = A.sub_ptr[blockIdx.x + 1];
    for (int q = q0; q < q1; ++q) {
        small_front<T, STRUCT, RPL>(A, q, member, smem_raw);
        __syncthreads();   // the front's shared memory is read out before the next front zeroes it
    }
}

// One Cholesky front of at most WARP_FRONT_F rows by one warp: assembled in its own shared-memory slice F (the
// lower triangle packed by columns: column j holds rows j .. f - 1 from offset j f - j (j - 1) / 2), then a row
// per lane in registers that shift down by one column a step. The arithmetic of every entry is small_front's
// with the front in registers, in the same order, so the results are its bit for bit. Batches of small systems
// have hundreds of thousands of such fronts; a launch of few fronts keeps the CTA kernel, whose 256 threads
// shorten each front's chain (lap2d 64^2 by the kernels before these: 1.04 against 1.35 ms a factorization). Fused subtrees keep the CTA
// kernel too: one warp per subtree was slower (1024 uneven systems: 6.79 against 5.93 ms).
//
// What bounds it: issue slots (half of them busy; a level of 488k fronts of about 12 rows 427 us, 703 with every
// front in 32 registers instead of 8, 16, 24 or 32 and the items by shuffles), then the dependent loads. 256
// systems of lap2d 96^2: factorization 5.8 -> 4.4 ms with this and the registers above. One warp for 16 members
// of a front, what they share loaded once: 1073 us for that level (neighbouring panels written far apart).
constexpr int WARP_FRONT_F = 32;
constexpr int WARP_FRONTS_PER_CTA = 4;
constexpr int WARP_FRONT_LEN = WARP_FRONT_F * (WARP_FRONT_F + 1) / 2;   // packed entries per warp
constexpr int64_t WARP_FRONT_MIN_LAUNCH = 4096;   // fronts x members of a launch for the warp kernel
constexpr int WARP_FRONT_U = 8;                   // columns of contributions in flight
template <typename T>
struct WarpItem {     // a column of a child's contribution: rows t .. mc - 1 at col, theirs in the front at sri
    const T* col;
    int sri, to;      // to: the packed place of the front's column | t << 16 | mc << 24
};
template <typename T>
__host__ __device__ constexpr int warp_front_bytes() {   // a warp's shared memory: its front, 32 items
    return WARP_FRONT_LEN * (int)sizeof(T) + 32 * (int)sizeof(WarpItem<T>);
}

// The assembled front F of f <= 8 G rows: factored in registers and written out. Rows above the diagonal and
// beyond the front hold whatever shared memory held: they reach no entry of the front.
template <typename T, int G>
__device__ __forceinline__ void warp_front_factor(const SmallArgs<T>& A, const SFront& fd, const int member, T* F) {
    const int f = fd.f, w = fd.w, m = f - w;
    const int lane = threadIdx.x & 31;
    T a[8 * G];
    const T* Fp = F + lane;
#pragma unroll
    for (int p = 0; p < 8 * G; ++p) {
        a[p] = *Fp;
        if (p + 1 < f) Fp += f - p - 1;
    }
    __syncwarp();
    // column j: lane's entry l, kept in F's place at the two buffers L[j & 1] (rows from j + 1 on)
    T* P = A.factor + (int64_t)member * A.factor_len + fd.panel + lane;
    int status = 0, j = 0;
    auto column = [&](auto n) {
        constexpr int N = decltype(n)::value;   // at least the columns that are left
        double r, root;
        if (!spd_pivot((double)__shfl_sync(0xffffffffu, a[0], j), A.eps, r, root)) {
            status = j + 1;
            return false;
        }
        T* L = F + (j & 1) * WARP_FRONT_F;
        const T l = a[0] * T(r);
        if (lane > j) L[lane - j - 1] = l;
        if (lane < f) *P = lane < j ? T(0) : lane == j ? T(root) : l;
        P += f;
        __syncwarp();
#pragma unroll
        for (int e = 0; e < N; e += 2) {
            using T2 = std::conditional_t<sizeof(T) == 8, double2, float2>;
            const T2 u = *reinterpret_cast<const T2*>(L + e);
            a[e] = fma(-l, u.x, a[e + 1]);
            if (e + 1 < N) a[e + 1] = fma(-l, u.y, a[e + 2]);
        }
        ++j;
        return true;
    };
    if constexpr (G >= 4)
        while (j < w && f - 1 - j > 23 && column(std::integral_constant<int, 31>())) {}
    if constexpr (G >= 3)
        while (status == 0 && j < w && f - 1 - j > 15 && column(std::integral_constant<int, 23>())) {}
    if constexpr (G >= 2)
        while (status == 0 && j < w && f - 1 - j > 7 && column(std::integral_constant<int, 15>())) {}
    while (status == 0 && j < w && column(std::integral_constant<int, 7>())) {}
    if (lane < NSTAT) {
        A.stats[((int64_t)member * A.ns + fd.s) * NSTAT + lane] =
            lane == ST_NPOS ? (status ? status - 1 : w) : lane == ST_INFO ? status : 0;
        if (lane == 0) A.finfo[(int64_t)member * A.ns + fd.s] = status;
    }
    if (fd.cb >= 0 && m > 0 && status == 0) {
        T* C = A.cb + (int64_t)member * A.cb_len + fd.cb + (lane - w);
#pragma unroll
        for (int e = 0; e < 8 * G; ++e) {
            if (lane >= w + e && lane < f) *C = a[e];
            C += m;
        }
    }
}

template <typename T>
__device__ __forceinline__ void warp_front_spd(const SmallArgs<T>& A, const int at, const int member, T* F,
                                               WarpItem<T>* items) {
    const SFront fd = A.sf[at];
    const int f = fd.f;
    const int lane = threadIdx.x & 31;
    auto column_at = [&](int j) { return j * f - ((j * (j + 1)) >> 1); };   // entry (i, j) is at column_at(j) + i
    const double* nz = A.nzval + (int64_t)member * A.nnz;
    const T* cbar = A.cb + (int64_t)member * A.cb_len;
    // the loads that do not depend on one another first
    int k = fd.am_begin + lane, code = 0, before = 0;
    double v0 = 0.0;
    if (k < fd.am_end) {
        code = A.maps.am_loc[k];
        before = k > fd.am_begin ? A.maps.am_loc[k - 1] : 0;
        v0 = nz[A.maps.am_src[k]];
    }
    auto fetch = [&](int e) {   // lane: item e + lane
        WarpItem<T> x{nullptr, 0, 255 << 16};
        if (e + lane < fd.nsri) {
            const uint32_t it = A.items[fd.sri_begin + e + lane];
            const SKid kid = A.kids[fd.kid_begin + ((it >> 8) & 0xffffu)];
            const int t = it & 0xffu;
            x = {cbar + kid.cb + (int64_t)t * kid.mc, fd.sri_begin + kid.sri,
                 column_at(it >> 24) | t << 16 | kid.mc << 24};
        }
        items[lane] = x;
    };
    if (fd.nsri > 0) fetch(0);
    for (int q = lane; q < (f * (f + 1)) / 2; q += 32) F[q] = T(0);
    __syncwarp();
    const int inv = 65536 / f + 1;   // loc / f = loc inv >> 16 for loc < f^2 <= 1024
    for (; k < fd.am_end; k += 32) {
        if (k != fd.am_begin + lane) {
            code = A.maps.am_loc[k];
            before = A.maps.am_loc[k - 1];
            v0 = nz[A.maps.am_src[k]];
        }
        if (before == code) continue;
        T acc = T(v0);
        for (int q = k + 1; q < fd.am_end && A.maps.am_loc[q] == code; ++q) acc += T(nz[A.maps.am_src[q]]);
        const int loc = (code > 0 ? code : -code) - 1;
        const int j = (loc * inv) >> 16, i = loc - j * f;
        // (an entry above the diagonal is never read by a Cholesky front)
        if (code > 0 && i >= j) F[column_at(j) + i] += acc;
        else if (code < 0 && j >= i) F[column_at(i) + j] += acc;
    }
    __syncwarp();
    // the children's columns by p mod 8, p and child: every entry's additions in child order
    for (int e = 0; e < fd.nsri; e += 32) {
        if (e > 0) {
            fetch(e);
            __syncwarp();
        }
        const int cnt = min(32, fd.nsri - e);
        for (int u0 = 0; u0 < cnt; u0 += WARP_FRONT_U) {
            T v[WARP_FRONT_U];
            int to[WARP_FRONT_U];
#pragma unroll
            for (int u = 0; u < WARP_FRONT_U; ++u) {
                const WarpItem<T> x = items[u0 + u];
                to[u] = -1;
                if (lane >= ((x.to >> 16) & 0xff) && lane < (x.to >> 24)) {
                    v[u] = x.col[lane];
                    to[u] = (x.to & 0xffff) + A.sri[x.sri + lane];
                }
            }
#pragma unroll
            for (int u = 0; u < WARP_FRONT_U; ++u) {
                if (to[u] >= 0) F[to[u]] += v[u];
                __syncwarp();
            }
        }
    }
    if (f <= 8) warp_front_factor<T, 1>(A, fd, member, F);
    else if (f <= 16) warp_front_factor<T, 2>(A, fd, member, F);
    else if (f <= 24) warp_front_factor<T, 3>(A, fd, member, F);
    else warp_front_factor<T, 4>(A, fd, member, F);
}

// Level launches of Cholesky fronts of at most 32 rows: one warp per front, WARP_FRONTS_PER_CTA per CTA.
template <typename T>
__global__ void __launch_bounds__(32 * WARP_FRONTS_PER_CTA) warp_front_kernel(SmallArgs<T> A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int wi = blockIdx.x * WARP_FRONTS_PER_CTA + (threadIdx.x >> 5);
    if (wi >= A.count) return;
    const int member = A.members ? A.members[blockIdx.y] : blockIdx.y;
    unsigned char* mine = smem_raw + (threadIdx.x >> 5) * warp_front_bytes<T>();
    warp_front_spd<T>(A, wi, member, reinterpret_cast<T*>(mine),
                      reinterpret_cast<WarpItem<T>*>(mine + WARP_FRONT_LEN * sizeof(T)));
}

size_t small_front_smem(int fmax, int elsize) {
    size_t ld = fmax | 1;
    size_t b = (ld * fmax * elsize + 15) & ~size_t(15);
    b += sizeof(SKid) * sf_kids(fmax) + 5 * sf_items(fmax);   // the staged kids, items and rows
    b += sizeof(double) * (2 * fmax + 2 * fmax);  // dd, ee (w <= f), lvec (2 f)
    b += sizeof(int) * (fmax + 16);               // lp, ctl
    b += fmax + 16;                               // kind
    return (b + 15) & ~size_t(15);
}

template <typename T>
cudaError_t launch_small(int structure, const SmallArgs<T>& a, int count, int nmembers, int fmax, cudaStream_t st) {
    const bool sub = a.sub_ptr != nullptr;
    SmallArgs<T> b = a;
    b.count = count;
    b.fmax = fmax;
    if (structure == STRUCT_SPD && fmax <= WARP_FRONT_F && !sub &&
        (int64_t)count * nmembers >= WARP_FRONT_MIN_LAUNCH) {   // a warp per front
        const size_t wsmem = (size_t)WARP_FRONTS_PER_CTA * warp_front_bytes<T>();
        dim3 wgrid((count + WARP_FRONTS_PER_CTA - 1) / WARP_FRONTS_PER_CTA, nmembers);
        warp_front_kernel<T><<<wgrid, 32 * WARP_FRONTS_PER_CTA, wsmem, st>>>(b);
        return cudaGetLastError();
    }
    size_t smem = small_front_smem(fmax, sizeof(T));
    const bool regs = structure == STRUCT_SPD && fmax <= 96;
    int threads = regs || fmax > 48 ? 256 : 128;
    dim3 grid(count, nmembers);
    auto go = [&](auto kern, auto sub_kern) {
        if (sub) sub_kern<<<grid, threads, smem, st>>>(b);
        else kern<<<grid, threads, smem, st>>>(b);
    };
    switch (structure) {
        case STRUCT_SPD:
            if (fmax <= 32) go(small_front_kernel<T, STRUCT_SPD, 1>, subtree_kernel<T, STRUCT_SPD, 1>);
            else if (fmax <= 64) go(small_front_kernel<T, STRUCT_SPD, 2>, subtree_kernel<T, STRUCT_SPD, 2>);
            else if (regs) go(small_front_kernel<T, STRUCT_SPD, 3>, subtree_kernel<T, STRUCT_SPD, 3>);
            else go(small_front_kernel<T, STRUCT_SPD, 0>, subtree_kernel<T, STRUCT_SPD, 0>);
            break;
        case STRUCT_S: go(small_front_kernel<T, STRUCT_S, 0>, subtree_kernel<T, STRUCT_S, 0>); break;
        default: go(small_front_kernel<T, STRUCT_G, 0>, subtree_kernel<T, STRUCT_G, 0>);
    }
    return cudaGetLastError();
}

// the opt-in shared-memory limit of every kernel with a dynamic allocation, set once at plan creation
// (outside any stream capture)
cudaError_t prepare_factor_kernels(int max_smem) {
    cudaError_t e = cudaSuccess;
    auto set = [&](const void* k) {
        if (e != cudaSuccess) return;
        cudaFuncAttributes fa;
        e = cudaFuncGetAttributes(&fa, k);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem - (int)fa.sharedSizeBytes);
    };
    set((const void*)small_front_kernel<double, STRUCT_SPD, 0>);
    set((const void*)small_front_kernel<double, STRUCT_SPD, 1>);
    set((const void*)small_front_kernel<double, STRUCT_SPD, 2>);
    set((const void*)small_front_kernel<double, STRUCT_SPD, 3>);
    set((const void*)small_front_kernel<double, STRUCT_S, 0>);
    set((const void*)small_front_kernel<double, STRUCT_G, 0>);
    set((const void*)small_front_kernel<float, STRUCT_SPD, 0>);
    set((const void*)small_front_kernel<float, STRUCT_SPD, 1>);
    set((const void*)small_front_kernel<float, STRUCT_SPD, 2>);
    set((const void*)small_front_kernel<float, STRUCT_SPD, 3>);
    set((const void*)small_front_kernel<float, STRUCT_S, 0>);
    set((const void*)small_front_kernel<float, STRUCT_G, 0>);
    set((const void*)subtree_kernel<double, STRUCT_SPD, 0>);
    set((const void*)subtree_kernel<double, STRUCT_SPD, 1>);
    set((const void*)subtree_kernel<double, STRUCT_SPD, 2>);
    set((const void*)subtree_kernel<double, STRUCT_SPD, 3>);
    set((const void*)subtree_kernel<double, STRUCT_S, 0>);
    set((const void*)subtree_kernel<double, STRUCT_G, 0>);
    set((const void*)subtree_kernel<float, STRUCT_SPD, 0>);
    set((const void*)subtree_kernel<float, STRUCT_SPD, 1>);
    set((const void*)subtree_kernel<float, STRUCT_SPD, 2>);
    set((const void*)subtree_kernel<float, STRUCT_SPD, 3>);
    set((const void*)subtree_kernel<float, STRUCT_S, 0>);
    set((const void*)subtree_kernel<float, STRUCT_G, 0>);
    set((const void*)warp_front_kernel<double>);
    set((const void*)warp_front_kernel<float>);
    return e;
}

template cudaError_t launch_small<double>(int, const SmallArgs<double>&, int, int, int, cudaStream_t);
template cudaError_t launch_small<float>(int, const SmallArgs<float>&, int, int, int, cudaStream_t);

// ---------------------------------------------------------------------------
// Column-owner assembly of large fronts (one warp per task).
// Storage of a large front: the panel (f x w, ld f) holds F[:, 0:w] -- for "S"
// both triangles of the fully-summed block -- ; "G" keeps F[j, i] (i > j, j < w)
// in the U^T panel at ufactor[panel + i + j f]; the contribution block
// F[w:f, w:f] lives at cb (ld m).
//
// A warp builds its column ASM_ROWS rows at a time in shared memory: the chunk
// starts at zero, takes the column's entries of A, then the rows of every
// child's contribution that land in it (the child's row-chunk table gives their
// range, relind being increasing) in the order of the column's extend-add list,
// and is written once. Every entry receives the same additions in the same
// order as a zero fill followed by accumulation in place, at one write of the
// entry instead of a write, a read and a write.
constexpr int ASM_WARPS = 8;
constexpr int ASM_KIDS = 8;   // child descriptors a warp keeps in shared memory per column

template <typename T>
struct AsmChild {
    const T* col;      // column t of the child's contribution block
    const int* ri;     // the child's relind
    const int* rc;     // the child's row-chunk starts
    int t, mc;
};

// buf[ri[q] - r0] += val(q) for q in [q0, q1) (lanes strided; the targets of one call are distinct);
// eight loads in flight per lane before the shared-memory updates
template <class T, class VAL>
__device__ __forceinline__ void chunk_add(T* buf, int r0, int q0, int q1, const int* ri, int lane, VAL val) {
    constexpr int U = ASM_ROWS / 32;
    for (int qb = q0 + lane; qb < q1; qb += 32 * U) {
        int pos[U];
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int q = qb + 32 * u;
            pos[u] = q < q1 ? ri[q] - r0 : -1;
            v[u] = q < q1 ? val(q) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (pos[u] >= 0) buf[pos[u]] = T((double)buf[pos[u]] + v[u]);
    }
}

template <typename T, int STRUCT>
__global__ void __launch_bounds__(ASM_WARPS * 32) assemble_large_kernel(LargeAsmArgs<T> A) {
    constexpr bool GEN = STRUCT == STRUCT_G;
    __shared__ T lbuf[ASM_WARPS][ASM_ROWS];
    __shared__ T ubuf[GEN ? ASM_WARPS : 1][GEN ? ASM_ROWS : 1];
    __shared__ AsmChild<T> kids[ASM_WARPS][ASM_KIDS];
    const int wid = threadIdx.x >> 5;
    const int task = blockIdx.x * ASM_WARPS + wid;
    const int lane = threadIdx.x & 31;
    if (task >= A.count) return;
    const int member = A.members ? A.members[blockIdx.y] : blockIdx.y;
    const ColTask ct = A.tasks[task];
    const DFront fd = A.maps.fronts[ct.front];
    const int f = fd.f, w = fd.w, m = f - w, p = ct.p;
    const bool panel = p < w;
    if (!panel && fd.cb < 0) return;
    const double* nz = A.nzval + (int64_t)member * A.nnz;
    const T* cbar = A.cb + (int64_t)member * A.cb_len;
    // the column indexed by front row: panel rows 0..f-1; contribution-block rows w..f-1 (from p for
    // the lower triangle of "SPD" and "S")
    T* lcol = panel ? A.factor + (int64_t)member * A.factor_len + fd.panel + (int64_t)p * f
                    : A.cb + (int64_t)member * A.cb_len + fd.cb + (int64_t)(p - w) * m - w;
    T* ucol = GEN && panel ? A.ufactor + (int64_t)member * A.factor_len + fd.panel + (int64_t)p * f : nullptr;
    const int rfirst = panel ? 0 : (GEN ? w : p);
    const int a0 = panel ? A.maps.amcol[fd.amcol_begin + p] : 0;
    const int a1 = panel ? A.maps.amcol[fd.amcol_begin + p + 1] : 0;
    const int e0 = A.maps.eacol[fd.eacol_begin + p], e1 = A.maps.eacol[fd.eacol_begin + p + 1];
    AsmChild<T>* kd = kids[wid];
    auto child = [&](int e) {
        AsmChild<T> k;
        const int c = A.maps.ea[2 * e];
        k.t = A.maps.ea[2 * e + 1];
        const DFront cd = A.maps.fronts[c];
        k.mc = cd.f - cd.w;
        k.col = cbar + cd.cb + (int64_t)k.t * k.mc;
        k.ri = A.maps.relind + cd.ri_begin;
        k.rc = A.maps.rchunk + cd.rc_begin;
        return k;
    };
    if (lane < ASM_KIDS && e0 + lane < e1) kd[lane] = child(e0 + lane);
    T* lb = lbuf[wid];
    T* ub = GEN ? ubuf[wid] : nullptr;
    __syncwarp();
    for (int r0 = rfirst; r0 < f;) {
        const int k = r0 / ASM_ROWS;
        const int r1 = min(f, (k + 1) * ASM_ROWS);
        const int len = r1 - r0;
        for (int i = lane; i < len; i += 32) {
            lb[i] = T(0);
            if (GEN && panel) ub[i] = T(0);
        }
        __syncwarp();
        // entries of A (runs of one location summed first, as the reference's assembly map lists them)
        for (int q = a0 + lane; q < a1; q += 32) {
            const int code = A.maps.am_loc[q];
            if (q > a0 && A.maps.am_loc[q - 1] == code) continue;
            const int row = (code > 0 ? code : -code) - 1 - p * f;
            if (row < r0 || row >= r1) continue;
            T acc = T(0);
            for (int z = q; z < a1 && A.maps.am_loc[z] == code; ++z) acc += T(nz[A.maps.am_src[z]]);
            if (code > 0) lb[row - r0] += acc;
            else ub[row - r0] += acc;
        }
        __syncwarp();
        for (int e = e0; e < e1; ++e) {
            const AsmChild<T> c = e - e0 < ASM_KIDS ? kd[e - e0] : child(e);
            const int lo = c.rc[k], hi = c.rc[k + 1];
            // column t of the child: its rows from the diagonal down land in column p; "G" contribution
            // block columns also take the rows above the diagonal (those below front row w are skipped by
            // the chunk bounds: they belong to the U^T panel)
            const int qb = (GEN && !panel) ? lo : max(lo, c.t);
            const T* col = c.col;
            chunk_add(lb, r0, qb, hi, c.ri, lane, [&](int q) { return (double)col[q]; });
            if (GEN && panel) {
                // row t of the child right of its diagonal: F[p, ri[jj]], the U^T panel column p
                const T* row = col - (int64_t)c.t * c.mc + c.t;
                const int64_t mcl = c.mc;
                chunk_add(ub, r0, max(lo, c.t + 1), hi, c.ri, lane, [&](int q) { return (double)row[q * mcl]; });
            }
            __syncwarp();
        }
        for (int i = lane; i < len; i += 32) {
            lcol[r0 + i] = lb[i];
            if (GEN && panel) ucol[r0 + i] = ub[i];
        }
        __syncwarp();
        r0 = r1;
    }
}

template <typename T>
cudaError_t launch_assemble_large(int structure, const LargeAsmArgs<T>& a, int nmembers, cudaStream_t st) {
    dim3 grid((a.count + ASM_WARPS - 1) / ASM_WARPS, nmembers);
    switch (structure) {
        case STRUCT_SPD: assemble_large_kernel<T, STRUCT_SPD><<<grid, ASM_WARPS * 32, 0, st>>>(a); break;
        case STRUCT_S: assemble_large_kernel<T, STRUCT_S><<<grid, ASM_WARPS * 32, 0, st>>>(a); break;
        default: assemble_large_kernel<T, STRUCT_G><<<grid, ASM_WARPS * 32, 0, st>>>(a);
    }
    return cudaGetLastError();
}

template cudaError_t launch_assemble_large<double>(int, const LargeAsmArgs<double>&, int, cudaStream_t);
template cudaError_t launch_assemble_large<float>(int, const LargeAsmArgs<float>&, int, cudaStream_t);

// ---------------------------------------------------------------------------
// Totals of the per-front statistics and the smallest failed factor column
// (reduce_stats! src/numeric/ldlt.jl:1276-1340, _cholesky_stats_kernel!
// src/numeric/factorize.jl:13-45): sums of integers, the same in any order.
__global__ void stats_kernel(StatsArgs A) {
    const int member = A.members ? A.members[blockIdx.y] : blockIdx.y;
    __shared__ int64_t red[NSTAT + 1][256];
    __shared__ bool last;
    int64_t acc[NSTAT] = {0, 0, 0, 0, 0, 0};
    int64_t best = INT64_MAX;
    const int64_t* S = A.stats + (int64_t)member * A.ns * NSTAT;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < A.ns; s += gridDim.x * blockDim.x) {
        for (int q = 0; q < NSTAT - 1; ++q) acc[q] += S[(int64_t)s * NSTAT + q];
        int64_t fi = S[(int64_t)s * NSTAT + ST_INFO];
        if (fi != 0) {
            acc[ST_INFO] += 1;
            best = min(best, (int64_t)A.super_ptr0[s] + fi - 1);
        }
    }
    for (int q = 0; q < NSTAT; ++q) red[q][threadIdx.x] = acc[q];
    red[NSTAT][threadIdx.x] = best;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if (threadIdx.x < h) {
            for (int q = 0; q < NSTAT; ++q) red[q][threadIdx.x] += red[q][threadIdx.x + h];
            red[NSTAT][threadIdx.x] = min(red[NSTAT][threadIdx.x], red[NSTAT][threadIdx.x + h]);
        }
        __syncthreads();
    }
    if (gridDim.x > 1) {   // the last CTA to finish adds every CTA's sums
        int64_t* part = A.part + (int64_t)member * STATS_MAX_CTAS * (NSTAT + 1);
        if (threadIdx.x == 0) {
            for (int q = 0; q <= NSTAT; ++q) part[blockIdx.x * (NSTAT + 1) + q] = red[q][0];
            __threadfence();
            last = atomicAdd(A.ticket + member, 1u) == gridDim.x - 1;
        }
        __syncthreads();
        if (!last) return;
        __threadfence();
        if (threadIdx.x <= NSTAT) {
            const int q = threadIdx.x;
            int64_t v = __ldcg(part + q);
            for (int c = 1; c < (int)gridDim.x; ++c) {
                const int64_t x = __ldcg(part + c * (NSTAT + 1) + q);
                v = q == NSTAT ? min(v, x) : v + x;
            }
            red[q][0] = v;
        }
        if (threadIdx.x == 0) A.ticket[member] = 0;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        for (int q = 0; q < NSTAT; ++q) A.totals[(int64_t)member * NSTAT + q] = red[q][0];
        int64_t b = red[NSTAT][0];
        A.info[member] = b == INT64_MAX ? 0 : (int64_t)A.perm0[b] + 1;  // original column, 1-based
    }
}

cudaError_t launch_stats(const StatsArgs& a, int nmembers, cudaStream_t st) {
    // one CTA took 0.42 ms over the 136 600 fronts of 256 uneven systems, at the end of a 1.7 ms factorization
    const int ctas = a.ns > 0 ? (a.ns + 2047) / 2048 : 1;
    stats_kernel<<<dim3(ctas < STATS_MAX_CTAS ? ctas : STATS_MAX_CTAS, nmembers), 256, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace sds
