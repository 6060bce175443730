// yk_cluster.cuh -- sums, barrier and remote shared memory of the solves that
// run inside one thread-block cluster (yk_cg_small.cu, yk_cg_eoc.cu).
#pragma once

#include <mutex>

#include "yk_ff.cuh"

namespace yk {

// f() once for each device of the process: a kernel's attributes hold for the device that
// was current.
template <typename F>
int once_per_device(F f)
{
    constexpr int kDevices = 64;
    static std::once_flag once[kDevices];
    static int value[kDevices];
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return f();
    std::call_once(once[dev], [&] { value[dev] = f(); });
    return value[dev];
}

// A sum in the precision it is carried: FP64, or float-float for FP32 vectors.
__device__ __forceinline__ double s_add(double a, double b) { return a + b; }
__device__ __forceinline__ FF s_add(FF a, FF b) { return ff_add(a, b); }
__device__ __forceinline__ double s_shfl(double a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
__device__ __forceinline__ FF s_shfl(FF a, int o) { return ff_shfl_xor(a, o); }
__device__ __forceinline__ double s_val(double a) { return a; }
__device__ __forceinline__ double s_val(FF a) { return (double)a.hi + (double)a.lo; }
__device__ __forceinline__ double s_of(double x, double) { return x; }
__device__ __forceinline__ FF s_of(double x, FF)
{
    const float hi = (float)x;
    return FF{hi, (float)(x - (double)hi)};
}
__device__ __forceinline__ FF s_of(float x, FF) { return FF{x, 0.f}; }
__device__ __forceinline__ FF s_of(FF x, FF) { return x; }
__device__ __forceinline__ double s_zero(double) { return 0.0; }
__device__ __forceinline__ FF s_zero(FF) { return FF{0.f, 0.f}; }

// Sums four values over the warp: lane l returns value l >> 3.
template <typename T>
__device__ __forceinline__ T warp_sum4(const T (&v)[4])
{
    const int lane = threadIdx.x & 31;
    const bool h = lane & 16, q = lane & 8;
    const T a0 = s_add(h ? v[2] : v[0], s_shfl(h ? v[0] : v[2], 16));
    const T a1 = s_add(h ? v[3] : v[1], s_shfl(h ? v[1] : v[3], 16));
    T c = s_add(q ? a1 : a0, s_shfl(q ? a0 : a1, 8));
    c = s_add(c, s_shfl(c, 4));
    c = s_add(c, s_shfl(c, 2));
    return s_add(c, s_shfl(c, 1));
}

__device__ __forceinline__ float warp_sum4(const float (&v)[4])
{
    const int lane = threadIdx.x & 31;
    const bool h = lane & 16, q = lane & 8;
    const unsigned full = 0xffffffffu;
    const float a0 = (h ? v[2] : v[0]) + __shfl_xor_sync(full, h ? v[0] : v[2], 16);
    const float a1 = (h ? v[3] : v[1]) + __shfl_xor_sync(full, h ? v[1] : v[3], 16);
    float c = (q ? a1 : a0) + __shfl_xor_sync(full, q ? a0 : a1, 8);
    c += __shfl_xor_sync(full, c, 4);
    c += __shfl_xor_sync(full, c, 2);
    return c + __shfl_xor_sync(full, c, 1);
}

__device__ __forceinline__ void cluster_barrier()
{
    __syncwarp();   // the aligned forms below want the warp converged
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Generic address of a shared-memory location of this CTA in CTA `rank`.
template <typename T>
__device__ __forceinline__ T* in_cta(T* p, unsigned rank)
{
    T* q;
    asm("mapa.u64 %0, %1, %2;" : "=l"(q) : "l"(p), "r"(rank));
    return q;
}

constexpr long long kClusterWaitCycles = 4000000000ll;   // about 2 s

// Shared-memory address of this CTA's location `p` in CTA `rank`.
__device__ __forceinline__ unsigned cta_addr(const void* p, unsigned rank)
{
    unsigned q;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(q) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return q;
}

// Asynchronous stores into another CTA that count their bytes on its mbarrier.
__device__ __forceinline__ void st_async(unsigned addr, float4 v, unsigned mbar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
                 "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(mbar)
                 : "memory");
}

__device__ __forceinline__ void st_async(unsigned addr, FF v, unsigned mbar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr), "f"(v.hi),
                 "f"(v.lo), "r"(mbar)
                 : "memory");
}

__device__ __forceinline__ void st_async(unsigned addr, double v, unsigned mbar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
                 "l"(__double_as_longlong(v)), "r"(mbar)
                 : "memory");
}

// words of 16 bytes
template <typename V>
__device__ __forceinline__ void st_async16(unsigned addr, const V& v, unsigned mbar)
{
    static_assert(sizeof(V) % 16 == 0, "words of 16 bytes");
    const float4* const p = reinterpret_cast<const float4*>(&v);
#pragma unroll
    for (int q = 0; q < (int)sizeof(V) / 16; ++q) st_async(addr + 16u * q, p[q], mbar);
}

__device__ __forceinline__ void mb_expect(unsigned mbar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}

// Waits for the mbarrier's phase.  A wait that gives up (about 2 s) says so in
// *dead, after which no wait of the CTA lasts and the solve ends.
__device__ __forceinline__ void mb_wait(unsigned mbar, unsigned parity, int* dead)
{
    auto done = [&] {
        unsigned ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(mbar), "r"(parity)
                     : "memory");
        return ok != 0;
    };
    if (done()) return;
    const long long t0 = clock64();
    while (!done())
        if (*(volatile int*)dead || clock64() - t0 > kClusterWaitCycles) {
            *(volatile int*)dead = 1;
            return;
        }
}

// The end of a solve: no CTA leaves while another may still store into it.  After a
// wait that gave up the CTAs no longer pass the same barriers (the one that gave up ends,
// the others may still be in a reliable update), so it tells every CTA, which ends its
// waits too, and those that know arrive at barriers until all have come here (*left
// counts them in each), then let the stores on their way arrive.  A CTA that gave up comes here
// with no more barriers behind it than any CTA's last one, so nobody leaves uninformed.
// Returns whether a wait gave up, and says so in *err.
__device__ __forceinline__ bool cluster_end(unsigned nc, int* dead, int* left, int* err)
{
    const unsigned tid = threadIdx.x;
    if (__syncthreads_or(*(volatile int*)dead) && tid < nc) *(volatile int*)in_cta(dead, tid) = 1;
    cluster_barrier();
    if (!*(volatile int*)dead) return false;
    if (tid < nc) atomicAdd(in_cta(left, tid), 1);
    const long long t0 = clock64();
    int more = 1;
    while (more) {
        cluster_barrier();
        more = __syncthreads_or(tid == 0 && *(volatile int*)left < (int)nc && clock64() - t0 < 4 * kClusterWaitCycles);
    }
    const long long t1 = clock64();
    while (clock64() - t1 < 200000) {
    }
    if (tid == 0) *err = YK_ETIMEOUT;
    return true;
}

}  // namespace yk
