/* Preloaded before libyukawa_gb300.so in a child process: calls of the CUDA
 * runtime that do more, or less, than they are asked to. */
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>

static void *real(const char *name)
{
    return dlsym(dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD), name);
}

static void *word;   /* the context's error word: what it last read as four bytes */
static int launches_to_go, status;

/* Before the n-th cluster or cooperative launch from now on the error word becomes
 * `st`, as if a wait of the kernel before it had given up. */
void fake_error(int n, int st)
{
    launches_to_go = n;
    status = st;
}

static int no_memory;

/* From now on (on) every device allocation fails, or none does (off). */
void fake_no_memory(int on) { no_memory = on; }

cudaError_t cudaMalloc(void **p, size_t n)
{
    cudaError_t (*f)(void **, size_t) = real("cudaMalloc");
    return no_memory ? cudaErrorMemoryAllocation : f(p, n);
}

cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, enum cudaMemcpyKind kind, cudaStream_t s)
{
    cudaError_t (*f)(void *, const void *, size_t, enum cudaMemcpyKind, cudaStream_t) = real("cudaMemcpyAsync");
    if (n == 4 && kind == cudaMemcpyDeviceToHost) word = (void *)src;
    return f(dst, src, n, kind, s);
}

static int device, cluster_attributes;

/* From now on the current device calls itself `d`. */
void fake_device(int d) { device = d; }

cudaError_t cudaGetDevice(int *d)
{
    *d = device;
    return cudaSuccess;
}

cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d)
{
    cudaError_t (*f)(int *, enum cudaDeviceAttr, int) = real("cudaDeviceGetAttribute");
    return f(v, a, d == device ? 0 : d);
}

/* Kernels opted in to clusters of more than eight blocks until now. */
int fake_cluster_attributes(void) { return cluster_attributes; }

cudaError_t cudaFuncSetAttribute(const void *fn, enum cudaFuncAttribute a, int v)
{
    cudaError_t (*f)(const void *, enum cudaFuncAttribute, int) = real("cudaFuncSetAttribute");
    cluster_attributes += a == cudaFuncAttributeNonPortableClusterSizeAllowed;
    return f(fn, a, v);
}

static int launches;

/* Kernels launched until now. */
int fake_launches(void) { return launches; }

cudaError_t __cudaLaunchKernel(void *k, dim3 grid, dim3 block, void **args, size_t smem, cudaStream_t s)
{
    cudaError_t (*f)(void *, dim3, dim3, void **, size_t, cudaStream_t) = real("__cudaLaunchKernel");
    ++launches;
    return f(k, grid, block, args, smem, s);
}

cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *cfg, const void *fn, void **args)
{
    ++launches;
    cudaError_t (*f)(const cudaLaunchConfig_t *, const void *, void **) = real("cudaLaunchKernelExC");
    if (launches_to_go > 0 && --launches_to_go == 0)
        cudaMemcpyAsync(word, &status, 4, cudaMemcpyHostToDevice, cfg->stream);
    return f(cfg, fn, args);
}
