// Wide LDLT / LU fronts of one-member plans in 32-column blocks (pivot_panel.cuh): the kernel and its launch.
//
// Compiled without floating-point contraction, like every unit that restates the reference's in-front
// arithmetic.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "common.cuh"
#include "kernels.cuh"

namespace sds {

// addresses of p and of the mbarrier in the cluster's CTA q
__device__ __forceinline__ void pp_remote(const void* p, int q, unsigned& ra) {
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(q));
}
// asynchronous stores into CTA q's shared memory; their bytes count into its mbarrier
template <typename V>
__device__ __forceinline__ void pp_x_store(V* p, int q, V v, unsigned long long* mbar) {
    unsigned ra, rm;
    pp_remote(p, q, ra);
    pp_remote(mbar, q, rm);
    if constexpr (sizeof(V) == 8) {
        unsigned long long b;
        memcpy(&b, &v, 8);
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(ra), "l"(b), "r"(rm)
                     : "memory");
    } else {
        static_assert(sizeof(V) == 4, "4 or 8 bytes");
        unsigned b;
        memcpy(&b, &v, 4);
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(ra), "r"(b), "r"(rm)
                     : "memory");
    }
}
__device__ __forceinline__ void pp_x_store2(double* p, int q, double x, double y, unsigned long long* mbar) {
    unsigned ra, rm;
    pp_remote(p, q, ra);
    pp_remote(mbar, q, rm);
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(ra), "d"(x), "d"(y),
                 "r"(rm)
                 : "memory");
}
__device__ __forceinline__ void pp_x_store2(float* p, int q, float x, float y, unsigned long long* mbar) {
    unsigned ra, rm;
    pp_remote(p, q, ra);
    pp_remote(mbar, q, rm);
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(ra), "f"(x), "f"(y),
                 "r"(rm)
                 : "memory");
}
__device__ __forceinline__ void pp_x_arm(unsigned long long* mbar, int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(mbar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ uint64_t pp_clock() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// The longest wait, and the status word that a wait sets when it gives up, which ends the others too (in shared
// memory: a wait that does not last needs neither in a register)
struct PanelLimit {
    int32_t* status;
    uint64_t ns;
};
// A waiting thread's look at the clock: the time of its first (t0 = 0: this is it), or 0: it gives up.
__device__ __forceinline__ uint64_t pp_waited(const PanelLimit& limit, uint64_t t0) {
    if (*(volatile int32_t*)limit.status != 0) return 0;
    const uint64_t now = pp_clock();
    if (t0 == 0) t0 = now;
    if (now - t0 < limit.ns) return t0;
    atomicExch(limit.status, 1);
    return 0;
}
// true: the phase is complete; false: the wait has given up, and nothing of the exchange may be used
__device__ __forceinline__ bool pp_x_wait(unsigned long long* mbar, int parity, const PanelLimit& limit) {
    const unsigned m = (unsigned)__cvta_generic_to_shared(mbar);
    uint64_t t0 = 0;
    for (unsigned spins = 0;; ++spins) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(m), "r"(parity)
            : "memory");
        if (done) return true;
        if ((spins & 63) == 63 && (t0 = pp_waited(limit, t0)) == 0) return false;
    }
}
__device__ __forceinline__ void pp_x_init(unsigned long long* mbar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// the first n threads of the CTA
__device__ __forceinline__ void pp_warps_barrier(int n) { asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory"); }

__device__ __forceinline__ void pp_store2(double* p, double x, double y) { *reinterpret_cast<double2*>(p) = make_double2(x, y); }
__device__ __forceinline__ void pp_store2(float* p, float x, float y) { *reinterpret_cast<float2*>(p) = make_float2(x, y); }
__device__ __forceinline__ void pp_load2(const double* p, double& x, double& y) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    x = v.x;
    y = v.y;
}
__device__ __forceinline__ void pp_load2(const float* p, float& x, float& y) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    x = v.x;
    y = v.y;
}

__device__ __forceinline__ void pp_cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// a front's CTAs meet in global memory; a wait that gives up clears *ok (shared)
__device__ __forceinline__ void pp_group_barrier(unsigned int* bar, unsigned int& epoch, int gs, const PanelLimit& limit, int* ok) {
    __syncthreads();
    if (threadIdx.x == 0) {
        epoch += gs;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        unsigned int v;
        uint64_t t0 = 0;
        for (unsigned spins = 0;; ++spins) {
            asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if ((int)(v - epoch) >= 0) break;
            if ((spins & 63) == 63 && (t0 = pp_waited(limit, t0)) == 0) {
                *ok = 0;
                break;
            }
            __nanosleep(20);
        }
    }
    __syncthreads();
}
// *gate (shared): n warps go through together, or none. One that waits too long closes it, which the last to
// arrive forestalls: the word decides, so that nobody stands alone at a barrier behind it. One lane calls it.
__device__ __forceinline__ bool pp_gate(int* gate, int n, const PanelLimit& limit) {
    constexpr int CLOSED = 1 << 30;
    for (int v = 0;;) {   // arrive, unless it is closed
        const int old = atomicCAS(gate, v, v + 1);
        if (old == v) break;
        if (old & CLOSED) return false;
        v = old;
    }
    uint64_t t0 = 0;
    for (unsigned spins = 0;; ++spins) {
        int v = *(volatile int*)gate;
        if (v == n) return true;
        if (v & CLOSED) return false;
        if ((spins & 63) == 63 && (t0 = pp_waited(limit, t0)) == 0)
            while (v < n) {   // close it, unless the last has come
                const int old = atomicCAS(gate, v, v | CLOSED);
                if (old == v) break;
                v = old;
            }
    }
}
// CTA q's copy of *p
__device__ __forceinline__ void pp_remote_set(int* p, int q, int v) {
    unsigned ra;
    pp_remote(p, q, ra);
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(ra), "r"(v) : "memory");
}

}  // namespace sds

#include "pivot_panel.cuh"

namespace sds {

template <typename T, int STRUCT>
__global__ void __launch_bounds__(PP_THREADS, 1) pivot_panel_kernel(LargePivotArgs<T> A, PanelGroups G) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PanelSmem<T>& S = *reinterpret_cast<PanelSmem<T>*>(smem_raw);
    if (threadIdx.x == 0) {
        pp_x_init(&S.mbar[0]);
        pp_x_init(&S.mbar[1]);
        S.dead = 0;
    }
    pp_cluster_barrier();
    unsigned xn = 0;
    for (int q = G.job_ptr[blockIdx.x]; q < G.job_ptr[blockIdx.x + 1]; ++q) {
        const PanelJob job = G.jobs[q];
        if (job.role != PANEL_IDLE) pp_front<T, STRUCT>(A, job, S, G, xn);
        // the cluster's CTAs start their next job, or leave, together: none writes into another's shared
        // memory before or after its front
        pp_cluster_barrier();
        // A wait gave up in this job, in any of them: the mbarriers hold what did not arrive, so no further job.
        // (A CTA that were a job ahead could set the word here only in its exchanges, which come behind a meeting
        // with this one.) Stores that nobody waits for may still be on their way: their CTAs stay a little.
        if (S.dead) {
            for (int i = 0; i < 100; ++i) __nanosleep(1000);
            return;
        }
    }
}

template <typename T, int STRUCT>
static cudaLaunchConfig_t panel_config(int grid, int csize, cudaStream_t st, cudaLaunchAttribute (&attr)[2]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(PP_THREADS);
    cfg.dynamicSmemBytes = sizeof(PanelSmem<T>);
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = csize;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeCooperative;
    attr[1].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cfg;
}

template <typename T>
cudaError_t launch_pivot_panel(int structure, const LargePivotArgs<T>& a, const PanelGroups& g, int grid, cudaStream_t st) {
    if (a.count == 0 || grid == 0) return cudaSuccess;
    cudaLaunchAttribute attr[2];
    if (structure == STRUCT_S) {
        const cudaLaunchConfig_t cfg = panel_config<T, STRUCT_S>(grid, g.csize, st, attr);
        return cudaLaunchKernelEx(&cfg, pivot_panel_kernel<T, STRUCT_S>, a, g);
    }
    const cudaLaunchConfig_t cfg = panel_config<T, STRUCT_G>(grid, g.csize, st, attr);
    return cudaLaunchKernelEx(&cfg, pivot_panel_kernel<T, STRUCT_G>, a, g);
}

template <typename T>
int pivot_panel_clusters(int structure, int csize) {
    cudaLaunchAttribute attr[2];
    int n = 0;
    cudaError_t e;
    if (structure == STRUCT_S) {
        cudaLaunchConfig_t cfg = panel_config<T, STRUCT_S>(csize, csize, nullptr, attr);
        cfg.numAttrs = 1;
        e = cudaOccupancyMaxActiveClusters(&n, pivot_panel_kernel<T, STRUCT_S>, &cfg);
    } else {
        cudaLaunchConfig_t cfg = panel_config<T, STRUCT_G>(csize, csize, nullptr, attr);
        cfg.numAttrs = 1;
        e = cudaOccupancyMaxActiveClusters(&n, pivot_panel_kernel<T, STRUCT_G>, &cfg);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

cudaError_t prepare_pivot_panel() {
    cudaError_t e = cudaSuccess;
    auto set = [&](const void* k, size_t smem) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    };
    set((const void*)pivot_panel_kernel<double, STRUCT_S>, sizeof(PanelSmem<double>));
    set((const void*)pivot_panel_kernel<double, STRUCT_G>, sizeof(PanelSmem<double>));
    set((const void*)pivot_panel_kernel<float, STRUCT_S>, sizeof(PanelSmem<float>));
    set((const void*)pivot_panel_kernel<float, STRUCT_G>, sizeof(PanelSmem<float>));
    return e;
}

template cudaError_t launch_pivot_panel<double>(int, const LargePivotArgs<double>&, const PanelGroups&, int, cudaStream_t);
template cudaError_t launch_pivot_panel<float>(int, const LargePivotArgs<float>&, const PanelGroups&, int, cudaStream_t);
template int pivot_panel_clusters<double>(int, int);
template int pivot_panel_clusters<float>(int, int);

}  // namespace sds
