// The panel pivot kernel's own code (csrc/numeric/pivot_panel.cuh) on the CPU, against the reference's in-front
// steps one after another.
//
// Every GPU thread is a fiber; warp operations, CTA barriers, cluster barriers, mbarriers and asynchronous
// remote stores are restated here. A scheduler picks the fibers at random, and a remote store reaches its CTA
// late: at a random moment or, over links chosen at random, only when nothing else can go on. So an exchange
// whose order rests on time and not on its protocol decides on stale values here, and the results differ. A
// wait that nothing can end, a store outside the front, its scratch or a CTA's shared memory, a misaligned
// pair, a result that differs in one bit from the serial steps: each is an error.
//
//   pivot_panel_check <seed> <cases>        random small fronts
//   pivot_panel_check <seed> <cases> giveup  a wait gives up at a random moment: every thread must come to its end
//   pivot_panel_check <seed> wide           clusters of 8 and 16 CTAs, blocks with and without the row copies
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <random>
#include <vector>

using std::isfinite;
using std::max;
using std::min;

// --- the machine ---------------------------------------------------------------------------------------------------
namespace emu {

struct Cluster;
struct Warp {
    unsigned long long v[2][32];
    long arrived = 0;
};
struct Cta {
    int bid = 0, rank = 0, left = 0;         // left: threads that have not returned
    long sync_arrived = 0, named_arrived = 0;
    char* smem = nullptr;
    size_t smem_size = 0;
    Cluster* cluster = nullptr;
};
struct Cluster {
    std::vector<Cta*> ctas;
    long arrived = 0;
};
struct Fiber {
    void* sp = nullptr;
    std::vector<char> stack;
    bool done = false;
    uint3 tid;
    Cta* cta;
    Warp* warp;
    long warp_ops = 0, sync_ops = 0, cluster_ops = 0, named_need = 0;
    // what it waits for: a count that reaches `target`, an mbarrier whose phase is no longer `parity`
    const long* count = nullptr;
    long target = 0;
    const struct Mbar* mbar = nullptr;
    int parity = 0;
    const int* gate = nullptr;               // a gate's word that reaches `target`, or is closed
    bool limited = false, expired = false;   // the wait has a limit; it has run out
    bool lingers = false;                    // until no store is on its way
    inline bool blocked() const;
};
struct Store {                                // a remote store on its way
    Cta* dst;
    size_t at, mbar;
    int bytes, link;
    unsigned long long v;
};

struct Mbar {
    int tx;
    short armed, phase;
    inline void check();
};
static_assert(sizeof(Mbar) == 8, "an mbarrier is 8 bytes");
Fiber* cur;
void* scheduler_sp;
std::vector<Fiber*> fibers;
std::vector<Store> flight;
inline bool Fiber::blocked() const {
    return !expired && ((count && *count < target) || (mbar && mbar->phase == parity) || (gate && *gate < target) ||
                        (lingers && !flight.empty()));
}
std::vector<char> slow;                       // per link (source, destination): held back until all else waits
long progress = 0;
std::mt19937 rng(1);
int threads_per_cta = 0;
long first_expiry = -1;                       // the progress at which a wait runs out, whatever it waits for (-1: never)
bool given_up = false;                        // ... and then the others, one after another

[[noreturn]] void die(const char* what) {
    printf("%s (CTA %d thread %u)\n", what, cur ? cur->cta->bid : -1, cur ? cur->tid.x : 0u);
    fflush(stdout);
    _Exit(2);
}
// saves the callee-saved registers and the stack pointer at *from, continues at `to` (x86-64)
extern "C" void emu_switch(void** from, void* to);
asm(R"(
.text
emu_switch:
    pushq %rbp
    pushq %rbx
    pushq %r12
    pushq %r13
    pushq %r14
    pushq %r15
    movq %rsp, (%rdi)
    movq %rsi, %rsp
    popq %r15
    popq %r14
    popq %r13
    popq %r12
    popq %rbx
    popq %rbp
    ret
)");
void yield() { emu_switch(&cur->sp, scheduler_sp); }
void wait_count(const long* count, long target, bool limited = false) {
    cur->count = count;
    cur->target = target;
    cur->limited = limited;
    while (cur->blocked()) yield();
    if (!limited) cur->count = nullptr;
}

unsigned long long* warp_sync(unsigned long long v) {
    Fiber* f = cur;
    const long op = f->warp_ops++;
    f->warp->v[op & 1][f->tid.x & 31] = v;
    f->warp->arrived++;
    progress++;
    wait_count(&f->warp->arrived, 32 * (op + 1));
    return f->warp->v[op & 1];
}
void cta_sync() {
    Fiber* f = cur;
    const long op = f->sync_ops++;
    f->cta->sync_arrived++;
    progress++;
    wait_count(&f->cta->sync_arrived, threads_per_cta * (op + 1));
}

void Mbar::check() {
    if (armed && tx == 0) {
        armed = 0;
        phase ^= 1;
        progress++;
    }
}

void deliver(size_t i) {
    const Store s = flight[i];
    flight[i] = flight.back();
    flight.pop_back();
    if (s.dst->left == 0) die("a store into the shared memory of a CTA that has left");
    memcpy(s.dst->smem + s.at, &s.v, s.bytes);
    Mbar* m = reinterpret_cast<Mbar*>(s.dst->smem + s.mbar);
    m->tx -= s.bytes;
    m->check();
    progress++;
}
size_t offset_of(const void* p, size_t bytes) {
    const size_t at = (const char*)p - cur->cta->smem;
    if (at + bytes > cur->cta->smem_size) die("a remote address outside shared memory");
    return at;
}
// one random round after another until every fiber has returned
void run() {
    const int nwarps = (int)fibers.size() / 32;
    int idle = 0;
    while (true) {
        bool any = false;
        const long before = progress;
        if (rng() % 64 == 0)
            for (auto& x : slow) x = rng() % 4 == 0;
        for (int w = 0; w < nwarps; ++w) {
            const bool skip = idle == 0 && rng() % 3 == 0;
            for (bool again = true; again;) {   // the warp until all its lanes wait
                again = false;
                for (int l = 0; l < 32; ++l) {
                    Fiber* f = fibers[32 * w + l];
                    if (f->done) continue;
                    any = true;
                    if (skip || f->blocked()) continue;
                    cur = f;
                    emu_switch(&scheduler_sp, f->sp);
                    again = true;
                }
            }
        }
        cur = nullptr;
        for (size_t i = flight.size(); i-- > 0;)
            if (!slow[flight[i].link] && rng() % 2) deliver(i);
        if (!any) break;
        if (first_expiry >= 0 && (given_up ? rng() % 4 == 0 : progress >= first_expiry)) {
            // a wait runs out: one at first, then some of those that wait and look at the status word
            std::vector<Fiber*> waiting;
            for (Fiber* f : fibers)
                if (!f->done && f->limited && f->blocked()) waiting.push_back(f);
            if (!waiting.empty()) {
                for (size_t n = given_up ? 1 + rng() % waiting.size() : 1; n-- > 0;) waiting[rng() % waiting.size()]->expired = true;
                given_up = true;
                progress++;
            }
        }
        if (progress != before) {
            idle = 0;
        } else if (++idle > 40 && flight.empty()) {
            die("every thread waits");
        } else if (idle > 1 && !flight.empty()) {   // what is held back, a part of it
            for (size_t n = 1 + rng() % flight.size(); n-- > 0;) deliver(rng() % flight.size());
        }
    }
    while (!flight.empty()) deliver(0);
}

}  // namespace emu

#undef __noinline__
#define __noinline__

// --- what the kernel's code calls ----------------------------------------------------------------------------------
static uint3 emu_thread() { return emu::cur->tid; }
#define threadIdx emu_thread()
static dim3 emu_block_dim(512);
#define blockDim emu_block_dim
#define __syncthreads emu::cta_sync
static void __syncwarp() { emu::warp_sync(0); }
static void __threadfence() {}
static unsigned __ballot_sync(unsigned, int p) {
    const unsigned long long* v = emu::warp_sync(p != 0);
    unsigned r = 0;
    for (int i = 0; i < 32; ++i) r |= v[i] ? 1u << i : 0u;
    return r;
}
template <class X>
static X __ldcg(const X* p) {
    return *p;
}
static int __ffs(unsigned x) { return __builtin_ffs((int)x); }
static int __popc(unsigned x) { return __builtin_popcount(x); }
static unsigned __reduce_max_sync(unsigned, unsigned x) {
    const unsigned long long* v = emu::warp_sync(x);
    unsigned r = 0;
    for (int i = 0; i < 32; ++i) r = max(r, (unsigned)v[i]);
    return r;
}
static unsigned __reduce_min_sync(unsigned, unsigned x) {
    const unsigned long long* v = emu::warp_sync(x);
    unsigned r = ~0u;
    for (int i = 0; i < 32; ++i) r = min(r, (unsigned)v[i]);
    return r;
}
static bool __any_sync(unsigned m, int p) { return __ballot_sync(m, p) != 0; }
static bool __all_sync(unsigned m, int p) { return __ballot_sync(m, p) == 0xffffffffu; }
template <class X>
static X emu_from_lane(X x, int lane) {
    unsigned long long b = 0;
    memcpy(&b, &x, sizeof(X));
    const unsigned long long* v = emu::warp_sync(b);
    X r;
    memcpy(&r, &v[lane & 31], sizeof(X));
    return r;
}
template <class X>
static X __shfl_xor_sync(unsigned, X x, int o) {
    return emu_from_lane(x, (int)(emu::cur->tid.x & 31) ^ o);
}
template <class X>
static X __shfl_sync(unsigned, X x, int lane) {
    return emu_from_lane(x, lane);
}
template <class To, class From>
static To emu_bits(From x) {
    To r;
    memcpy(&r, &x, sizeof(To));
    return r;
}
static long long __double_as_longlong(double d) { return emu_bits<long long>(d); }
static double __longlong_as_double(long long b) { return emu_bits<double>(b); }
static unsigned __float_as_uint(float d) { return emu_bits<unsigned>(d); }
static float __uint_as_float(unsigned b) { return emu_bits<float>(b); }
static int atomicAdd(int* p, int v) {
    const int old = *p;
    *p += v;
    return old;
}

namespace sds {

template <typename V>
static void pp_x_store(V* p, int q, V v, unsigned long long* mbar) {
    emu::Cta* c = emu::cur->cta;
    if (q < 0 || q >= (int)c->cluster->ctas.size()) emu::die("a remote store to a CTA that is not in the cluster");
    emu::Store s{c->cluster->ctas[q], emu::offset_of(p, sizeof(V)), emu::offset_of(mbar, 8), (int)sizeof(V),
                 c->rank * 16 + q, 0};
    memcpy(&s.v, &v, sizeof(V));
    emu::flight.push_back(s);
    emu::progress++;
}
template <typename V>
static void emu_aligned(const V* p) {
    if ((uintptr_t)p % (2 * sizeof(V))) emu::die("a misaligned pair");
}
template <typename V>
static void pp_x_store2(V* p, int q, V x, V y, unsigned long long* mbar) {
    emu_aligned(p);
    pp_x_store(p, q, x, mbar);
    pp_x_store(p + 1, q, y, mbar);
}
static emu::Mbar* emu_mbar(unsigned long long* mbar) { return reinterpret_cast<emu::Mbar*>(mbar); }
static void pp_x_arm(unsigned long long* mbar, int bytes) {
    emu::Mbar* m = emu_mbar(mbar);
    if (m->armed) emu::die("an mbarrier armed twice");
    m->tx += bytes;
    m->armed = 1;
    m->check();
    emu::progress++;
}
struct PanelLimit {
    int32_t* status;
    uint64_t ns;
};
// the end of a wait with a limit: true, what it waited for has come
static bool emu_end(int32_t* status, bool come) {
    emu::Fiber* f = emu::cur;
    f->limited = false;
    f->count = nullptr;
    f->mbar = nullptr;
    const bool gave_up = f->expired && !come;
    f->expired = false;
    if (gave_up) *status = 1;
    return !gave_up;
}
static bool pp_x_wait(unsigned long long* mbar, int parity, const PanelLimit& limit) {
    emu::Fiber* f = emu::cur;
    f->mbar = emu_mbar(mbar);
    f->parity = parity;
    f->limited = true;
    while (f->blocked()) emu::yield();
    return emu_end(limit.status, f->mbar->phase != parity);
}
// the first n threads of the CTA
static void pp_warps_barrier(int n) {
    emu::Fiber* f = emu::cur;
    f->cta->named_arrived++;
    f->named_need += n;   // the same n for every arrival of one barrier
    emu::progress++;
    emu::wait_count(&f->cta->named_arrived, f->named_need);
}
template <typename V>
static void pp_store2(V* p, V x, V y) {
    emu_aligned(p);
    p[0] = x;
    p[1] = y;
}
template <typename V>
static void pp_load2(const V* p, V& x, V& y) {
    emu_aligned(p);
    x = p[0];
    y = p[1];
}
static void pp_cluster_barrier() {
    emu::Fiber* f = emu::cur;
    emu::Cluster* c = f->cta->cluster;
    const long op = f->cluster_ops++;
    c->arrived++;
    emu::progress++;
    emu::wait_count(&c->arrived, (long)c->ctas.size() * emu::threads_per_cta * (op + 1));
}
static long emu_group_arrived;
static void pp_group_barrier(unsigned*, unsigned& epoch, int gs, const PanelLimit& limit, int* ok) {
    emu::cta_sync();
    if (emu::cur->tid.x == 0) {
        epoch += gs;
        emu_group_arrived++;
        emu::progress++;
        emu::wait_count(&emu_group_arrived, epoch, true);
        if (!emu_end(limit.status, emu_group_arrived >= (long)epoch)) *ok = 0;
    }
    emu::cta_sync();
}
static bool pp_gate(int* gate, int n, const PanelLimit& limit) {
    constexpr int CLOSED = 1 << 30;
    if (*gate & CLOSED) return false;
    ++*gate;
    emu::progress++;
    emu::cur->limited = true;
    emu::cur->gate = gate;
    emu::cur->target = n;
    while (emu::cur->blocked()) emu::yield();
    emu::cur->gate = nullptr;
    if (!emu_end(limit.status, *gate >= n)) *gate |= CLOSED;   // (an n that was reached stays)
    return *gate == n;
}
static void pp_remote_set(int* p, int q, int v) {
    emu::Cta* d = emu::cur->cta->cluster->ctas[q];
    if (d->left == 0) emu::die("a store into the shared memory of a CTA that has left");
    *reinterpret_cast<int*>(d->smem + emu::offset_of(p, sizeof(int))) = v;
}

}  // namespace sds

#include "../../sparsedirectsolver.jl_b200/csrc/numeric/pivot_panel.cuh"

using namespace sds;

// --- the steps one after another -----------------------------------------------------------------------------------
struct SerialTeam {
    int rank = 0;
    static constexpr int size = 1;
    double reduce_jmax(double v) const { return v; }
    void reduce_argmax(double&, int&) const {}
};

struct Pivots {
    std::vector<int> lp;
    std::vector<signed char> kind;
    std::vector<double> d, e;
    int64_t st[NSTAT] = {};
};

struct Options {
    int pivot = PIVOT_BK, lu_pivot = 1;
    double u = 0.01, eps = 1e-13;
};

template <typename T, int STRUCT>
static Pivots serial(T* P, T* U, int f, int w, const Options& o) {
    constexpr bool GEN = STRUCT == STRUCT_G;
    GlobalStore<T, GEN> F{P, U, f, w};
    const SerialTeam tm;
    Pivots R;
    R.lp.resize(w);
    R.kind.resize(w);
    R.d.resize(w);
    R.e.assign(w, 0.0);
    if (!GEN)
        for (int j = 0; j < w; ++j)
            for (int i = j + 1; i < w; ++i) P[j + (int64_t)i * f] = P[i + (int64_t)j * f];
    for (int q = 0; q < w; ++q) R.lp[q] = q;
    auto perturb = [&](int k, int col) {   // the 1x1 pivot of column k
        double dk = F.get(k, k);
        R.kind[k] = KIND_1X1;
        if (!(fabs(dk) >= o.eps) || dk == 0.0) {
            if (dk == 0.0) R.st[ST_NZERO]++;
            dk = perturb_sign_of(dk, 0) * o.eps;
            R.kind[k] = KIND_PERTURBED;
            R.st[ST_NPERT]++;
            if (dk == 0.0 && R.st[ST_INFO] == 0) R.st[ST_INFO] = col + 1;
        }
        F.at(k, k) = T(dk);
        R.d[k] = dk;
        return dk;
    };
    std::vector<double> l1(f), l2(f);
    for (int k = 0; k < w;) {
        if (GEN) {
            const int r = o.lu_pivot ? lu_choose_row(F, k, w, o.u, tm) : k;
            if (r != k) {
                for (int j = 0; j < f; ++j) std::swap(F.at(k, j), F.at(r, j));
                std::swap(R.lp[k], R.lp[r]);
            }
            const T t = T(perturb(k, k));
            for (int j = k + 1; j < f; ++j) {
                const T fk = F.at(k, j);
                for (int i = k + 1; i < (j < w ? f : w); ++i) {
                    const T l = F.at(i, k) / t, pr = l * fk;
                    F.at(i, j) = F.at(i, j) - pr;
                }
            }
            for (int i = k + 1; i < f; ++i) F.at(i, k) /= t;
            for (int j = k + 1; j < f; ++j) F.at(k, j) /= t;
            k++;
            continue;
        }
        int c, r;
        choose_pivot(F, k, w, o.pivot, o.u, o.eps, tm, c, r);
        const int p = r < 0 ? k : k + 1, q = r < 0 ? c : r;
        if (p != q) {
            for (int i = 0; i < f; ++i) std::swap(F.at(i, p), F.at(i, q));
            for (int j = 0; j < w; ++j) std::swap(F.at(p, j), F.at(q, j));
            std::swap(R.lp[p], R.lp[q]);
        }
        if (r < 0) {
            const double dk = perturb(k, R.lp[k]);
            if (dk > 0) R.st[ST_NPOS]++;
            else if (dk < 0) R.st[ST_NNEG]++;
            for (int i = k + 1; i < f; ++i) l1[i] = F.get(i, k) / dk;
            for (int j = k + 1; j < w; ++j) {
                const T fk = F.at(k, j);
                for (int i = k + 1; i < f; ++i) {
                    const T pr = T(l1[i]) * fk;
                    F.at(i, j) = F.at(i, j) - pr;
                }
            }
            for (int i = k + 1; i < f; ++i) F.at(i, k) = T(l1[i]);
            k++;
            continue;
        }
        const double a = F.get(k, k), b = F.get(k + 1, k), c2 = F.get(k + 1, k + 1), det = a * c2 - b * b;
        const double e11 = c2 / det, e12 = -b / det, e21 = -b / det, e22 = a / det;
        R.st[ST_N2X2]++;
        if (det < 0) {
            R.st[ST_NPOS]++;
            R.st[ST_NNEG]++;
        } else {
            R.st[a > 0 ? ST_NPOS : ST_NNEG] += 2;
        }
        for (int i = k + 2; i < f; ++i) {
            const double x1 = F.get(i, k), x2 = F.get(i, k + 1);
            l1[i] = x1 * e11 + x2 * e21;
            l2[i] = x1 * e12 + x2 * e22;
        }
        R.d[k] = a;
        R.d[k + 1] = c2;
        R.e[k] = b;
        R.kind[k] = KIND_2X2_FIRST;
        R.kind[k + 1] = KIND_2X2_SECOND;
        for (int j = k + 2; j < w; ++j) {
            const T f1 = F.at(k, j), f2 = F.at(k + 1, j);
            for (int i = k + 2; i < f; ++i) {
                const T p1 = T(l1[i]) * f1, p2 = T(l2[i]) * f2, s = p1 + p2;
                F.at(i, j) = F.at(i, j) - s;
            }
        }
        for (int i = k + 2; i < f; ++i) {
            F.at(i, k) = T(l1[i]);
            F.at(i, k + 1) = T(l2[i]);
        }
        F.at(k + 1, k) = T(0);
        k += 2;
    }
    for (int j = 0; j < w; ++j)
        for (int i = 0; i <= j; ++i) {
            if (i == j) {
                P[i + (int64_t)j * f] = 1;
                if (GEN) U[i + (int64_t)j * f] = 1;
            } else if (!GEN) {
                P[i + (int64_t)j * f] = 0;
            }
        }
    return R;
}

// --- one front, both ways ------------------------------------------------------------------------------------------
enum Values { POSITIVE, ZERO_DIAGONALS, SMALL_INTEGERS, MANY_ZEROS, WEAK_DIAGONAL, FAR_PARTNERS, NVALUES };

template <typename T>
static bool same(const T& a, const T& b) {
    return a == b || (a != a && b != b);
}

static std::function<void()> thread_body;
static void thread_start() {
    thread_body();
    emu::cur->done = true;
    emu::cur->cta->left--;
    emu::progress++;
    emu::yield();
}

template <typename T, int STRUCT>
static bool check(int f, int w, int C, int nclusters, int values, const Options& o, unsigned seed, bool give_up) {
    constexpr bool GEN = STRUCT == STRUCT_G;
    std::mt19937 g(seed);
    std::normal_distribution<double> normal;
    auto value = [&]() -> double {
        if (values == SMALL_INTEGERS) return double(int(g() % 5) - 2);
        if (values == MANY_ZEROS) return g() % 3 ? 0.0 : normal(g);
        return (values == FAR_PARTNERS ? 0.01 : 1.0) * normal(g);
    };
    const int64_t len = (int64_t)f * w, GUARD = 4096;
    std::vector<T> P0(len + 2 * GUARD, T(777)), U0(len + 2 * GUARD, T(777));
    for (int j = 0; j < w; ++j)
        for (int i = 0; i < f; ++i) {
            T& p = P0[GUARD + i + (int64_t)j * f];
            p = T(i >= j ? value() : 0);
            U0[GUARD + i + (int64_t)j * f] = T(i > j ? value() : 0);
            if (i == j) {
                double d = value();
                if (values == POSITIVE) d = fabs(d) + 2 * sqrt((double)f);
                if (values == ZERO_DIAGONALS && i % 2) d = 0;
                if (values == WEAK_DIAGONAL || values == FAR_PARTNERS) d *= 1e-3;
                p = T(d);
            }
            if (values == FAR_PARTNERS && i < w && i == j + w / 2) p = T(1 + 0.1 * normal(g));
        }
    std::vector<T> P1 = P0, U1 = U0, P2 = P0, U2 = U0;
    const Pivots want = serial<T, STRUCT>(&P1[GUARD], &U1[GUARD], f, w, o);

    DFront fd{};
    fd.f = f;
    fd.w = w;
    const int32_t list[1] = {0};
    const int64_t scr_off[1] = {0};
    const int PAD = 32;
    std::vector<double> scratch(panel_scratch_len(f, w) + 2 * PAD, 777.0), d(2 * w);
    std::vector<int32_t> piv(w), perm(w, 0);
    std::vector<int8_t> kind(w);
    std::vector<int64_t> st(NSTAT, -1);
    int32_t finfo = -1, status = 0;
    unsigned bar = 0;
    LargePivotArgs<T> A{};
    A.fronts = &fd;
    A.list = list;
    A.count = 1;
    A.factor = &P2[GUARD];
    A.ufactor = &U2[GUARD];
    A.scratch = scratch.data() + PAD;
    A.scr_off = scr_off;
    A.d = d.data();
    A.piv = piv.data();
    A.kind = kind.data();
    A.stats = st.data();
    A.finfo = &finfo;
    A.perm = perm.data();
    A.n = w;
    A.ns = 1;
    A.pivot = o.pivot;
    A.lu_pivot = o.lu_pivot;
    A.u = o.u;
    A.eps = o.eps;

    const int ncta = C * nclusters;
    std::vector<emu::Cluster> clusters(nclusters);
    std::vector<emu::Cta> ctas(ncta);
    std::vector<emu::Warp> warps(ncta * PP_WARPS);
    std::vector<std::vector<char>> smem(ncta);
    std::vector<PanelJob> jobs(ncta);
    emu::threads_per_cta = PP_THREADS;
    emu::slow.assign(16 * 16, 0);
    for (int b = 0; b < ncta; ++b) {
        emu::Cta& c = ctas[b];
        smem[b].assign(sizeof(PanelSmem<T>) + 32, (char)0x7f);
        c.smem = (char*)(((uintptr_t)smem[b].data() + 15) & ~(uintptr_t)15);
        c.smem_size = sizeof(PanelSmem<T>);
        c.bid = b;
        c.rank = b % C;
        c.left = PP_THREADS;
        c.cluster = &clusters[b / C];
        c.cluster->ctas.push_back(&c);
        auto* S = reinterpret_cast<PanelSmem<T>*>(c.smem);
        S->mbar[0] = S->mbar[1] = 0;
        S->dead = 0;
        if (C == 1) jobs[b] = {b == 0 ? PANEL_SINGLE : PANEL_IDLE, 0, 0, 1};
        else jobs[b] = {b < C ? PANEL_LEAD : PANEL_HELP, 0, b, ncta};
    }
    thread_body = [&] {
        emu::Cta* c = emu::cur->cta;
        const PanelJob job = jobs[c->bid];
        const PanelGroups G{jobs.data(), nullptr, &bar, &status, 0, C};
        PanelSmem<T>& S = *reinterpret_cast<PanelSmem<T>*>(c->smem);
        unsigned xn = 0;
        if (job.role != PANEL_IDLE) pp_front<T, STRUCT>(A, job, S, G, xn);
        pp_cluster_barrier();
        emu::cur->lingers = S.dead != 0;
        while (emu::cur->blocked()) emu::yield();
        emu::cur->lingers = false;
    };
    for (auto* x : emu::fibers) delete x;
    emu::fibers.clear();
    for (int b = 0; b < ncta; ++b)
        for (int t = 0; t < PP_THREADS; ++t) {
            auto* x = new emu::Fiber;
            x->stack.resize(24576);
            x->tid = {(unsigned)t, 0, 0};
            x->cta = &ctas[b];
            x->warp = &warps[b * PP_WARPS + t / 32];
            // six registers and the return address; the stack is aligned as after a call
            void** top = (void**)(((uintptr_t)x->stack.data() + x->stack.size()) & ~(uintptr_t)15) - 1;
            *--top = (void*)thread_start;
            x->sp = top - 6;
            emu::fibers.push_back(x);
        }
    emu_group_arrived = 0;
    emu::given_up = false;
    emu::first_expiry = give_up ? emu::progress + (long)(g() % (60000 + 100 * w * ncta)) : -1;
    emu::run();

    bool ok = true;
    auto fail = [&](const char* what, int64_t at) {
        if (ok) printf("%s differs at %ld: ", what, (long)at);
        ok = false;
    };
    if (give_up && status) {   // the panels are what they are; nothing around them has changed
        for (int64_t q = 0; q < GUARD; ++q)
            for (auto* v : {&P2, &U2})
                if ((*v)[q] != T(777) || (*v)[len + GUARD + q] != T(777)) fail("a guard", q);
        for (int i = 0; i < PAD; ++i)
            if (scratch[i] != 777.0 || scratch[scratch.size() - 1 - i] != 777.0) fail("the scratch's guard", i);
        printf("%s %s FP%zu f %d w %d, %d clusters of %d: given up\n", ok ? "ok" : "FAIL", GEN ? "LU" : "LDLT", 8 * sizeof(T), f, w,
               nclusters, C);
        fflush(stdout);
        return ok;
    }
    if (status) fail("the status word", 0);
    for (int64_t q = 0; q < len + 2 * GUARD; ++q) {
        if (!same(P1[q], P2[q])) fail("the panel", q - GUARD);
        if (GEN && !same(U1[q], U2[q])) fail("the U^T panel", q - GUARD);
    }
    for (int i = 0; i < PAD; ++i)
        if (scratch[i] != 777.0 || scratch[scratch.size() - 1 - i] != 777.0) fail("the scratch's guard", i);
    for (int q = 0; q < w; ++q)
        if (piv[q] != want.lp[q] + 1 || kind[q] != want.kind[q] || !same(d[q], want.d[q]) ||
            (!GEN && !same(d[w + q], want.e[q])))
            fail("the pivot", q);
    for (int q = 0; q < NSTAT; ++q)
        if (st[q] != want.st[q]) fail("the statistics", q);
    if (finfo != want.st[ST_INFO]) fail("the info", 0);
    int swaps = 0;
    for (int q = 0; q < w; ++q) swaps += want.lp[q] != q;
    printf("%s %s FP%zu f %d w %d, %d clusters of %d, values %d pivot %d %d u %g eps %g: %d interchanges, %ld 2x2, %ld perturbed\n",
           ok ? "ok" : "FAIL", GEN ? "LU" : "LDLT", 8 * sizeof(T), f, w, nclusters, C, values, o.pivot, o.lu_pivot, o.u, o.eps,
           swaps, (long)want.st[ST_N2X2], (long)want.st[ST_NPERT]);
    fflush(stdout);
    return ok;
}

static bool check_any(bool gen, bool fp32, int f, int w, int C, int nclusters, int values, const Options& o, unsigned seed,
                      bool give_up = false) {
    if (gen) return fp32 ? check<float, STRUCT_G>(f, w, C, nclusters, values, o, seed, give_up)
                         : check<double, STRUCT_G>(f, w, C, nclusters, values, o, seed, give_up);
    return fp32 ? check<float, STRUCT_S>(f, w, C, nclusters, values, o, seed, give_up)
                : check<double, STRUCT_S>(f, w, C, nclusters, values, o, seed, give_up);
}

int main(int argc, char** argv) {
    const unsigned seed = argc > 1 ? atoi(argv[1]) : 1;
    const bool give_up = argc > 3 && !strcmp(argv[3], "giveup");
    std::mt19937 g(seed);
    emu::rng.seed(seed);
    auto pick = [&](std::initializer_list<double> v) { return v.begin()[g() % v.size()]; };
    bool ok = true;
    if (argc > 2 && !strcmp(argv[2], "wide")) {
        // the copies need 15 row warps at most: 480 C rows; values that reject pivots and reach out of the block
        struct { int f, w, C; } sizes[] = {{300, 36, 8}, {950, 34, 2}, {1000, 34, 2}, {700, 34, 16}, {470, 20, 16}};
        for (auto& s : sizes)
            for (int gen = 0; gen < 2; ++gen) {
                Options o;
                o.u = pick({0.01, 0.5, 1.0});
                ok &= check_any(gen, g() % 2, s.f, s.w, s.C, 1, gen ? WEAK_DIAGONAL : (int)(g() % NVALUES), o, g());
            }
    } else {
        for (int n = argc > 2 ? atoi(argv[2]) : 20, q = 0; q < n; ++q) {
            const int w = 1 + g() % (q % 3 == 0 ? 40 : 110), f = w + (g() % 4 == 0 ? 0 : g() % 200);
            const int C = give_up ? (int)pick({2, 4, 8}) : (int)pick({1, 2, 4, 8}), nclusters = C == 1 || C == 8 ? 1 : 1 + g() % 2;
            Options o;
            o.u = pick({0.01, 0.1, 0.5, 0.9, 1.0});
            o.eps = pick({1e-13, 1e-13, 0.0, 0.5});
            const bool gen = g() % 3 == 0;
            if (!gen) o.pivot = (int)pick({(double)PIVOT_BK, (double)PIVOT_BK, (double)PIVOT_BK, (double)PIVOT_NONE, (double)PIVOT_DIAGONAL});
            else o.lu_pivot = g() % 4 != 0;
            ok &= check_any(gen, g() % 3 == 0, f, w, C, nclusters, g() % NVALUES, o, g(), give_up);
        }
    }
    printf(ok ? "all ok\n" : "FAILED\n");
    return !ok;
}
