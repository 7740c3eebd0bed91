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
// a wait of some seconds at most, then the status word (which later waits do not outlast)
__device__ __forceinline__ void pp_x_wait(unsigned long long* mbar, int parity, int32_t* status) {
    const unsigned m = (unsigned)__cvta_generic_to_shared(mbar);
    for (unsigned spins = 0;; ++spins) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(m), "r"(parity)
            : "memory");
        if (done) return;
        if ((spins & 1023) == 1023 && *(volatile int32_t*)status != 0) return;
        if (spins > (1u << 24)) {
            atomicExch(status, 1);
            return;
        }
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

// one value from global into shared memory in the background (zero when not valid)
__device__ __forceinline__ void pp_fetch(double* s, const double* g, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g),
                 "r"(valid ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void pp_fetch(float* s, const float* g, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g),
                 "r"(valid ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void pp_fetch_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void pp_cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// a front's CTAs meet in global memory; a wait of about two seconds gives up, records the status word and
// clears *ok (shared), as does a status word that is already set
__device__ __forceinline__ void pp_group_barrier(unsigned int* bar, unsigned int& epoch, int gs, int32_t* status, int* ok) {
    __syncthreads();
    if (threadIdx.x == 0) {
        epoch += gs;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        unsigned int v;
        for (long spins = 0;; ++spins) {
            asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if ((int)(v - epoch) >= 0) break;
            if ((spins & 255) == 255 && *(volatile int32_t*)status != 0) {
                *ok = 0;
                break;
            }
            if (spins > (1L << 25)) {
                atomicExch(status, 1);
                *ok = 0;
                break;
            }
            __nanosleep(20);
        }
    }
    __syncthreads();
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
    }
    pp_cluster_barrier();
    unsigned xn = 0;
    for (int q = G.job_ptr[blockIdx.x]; q < G.job_ptr[blockIdx.x + 1]; ++q) {
        const PanelJob job = G.jobs[q];
        if (job.role != PANEL_IDLE) pp_front<T, STRUCT>(A, job, S, G.csize, G.bar, G.status, xn);
        // the cluster's CTAs start their next job, or leave, together: none writes into another's shared
        // memory before or after its front
        pp_cluster_barrier();
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
