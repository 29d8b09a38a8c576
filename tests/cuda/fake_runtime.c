/* A stand-in for the CUDA runtime, for tests of the host code without a GPU.
 * Loaded before the library (RTLD_GLOBAL), its definitions are the ones that the
 * library's calls reach: nothing runs on a device, "device" memory is host memory,
 * and the function attributes, launches and copies are written to a log, one per line:
 *   attr <kernel> <attribute> <value>
 *   launch <kernel> <grid x> <y> <z> <threads per block> <dynamic shared memory>
 *   copy <bytes> <kind>
 * A kernel is named as the compiler registers it (mangled). */
#include <cuda_runtime_api.h>
#include <pthread.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define MAX_KERNELS 65536
static const void *funcs[MAX_KERNELS];
static const char *names[MAX_KERNELS];
static int n_kernels;
static char text[1 << 24];
static size_t used;

const char *fake_log(void) { return text; }
void fake_reset(void) { text[used = 0] = 0; }

static void note(const char *fmt, ...)
{
    static pthread_mutex_t lock = PTHREAD_MUTEX_INITIALIZER;   /* the library's copies run on several threads */
    va_list ap;
    va_start(ap, fmt);
    pthread_mutex_lock(&lock);
    const int n = vsnprintf(text + used, sizeof(text) - used, fmt, ap);
    if (n > 0 && used + (size_t)n < sizeof(text)) used += (size_t)n;
    pthread_mutex_unlock(&lock);
    va_end(ap);
}
static const char *name_of(const void *f)
{
    for (int k = 0; k < n_kernels; ++k)
        if (funcs[k] == f) return names[k];
    return "?";
}
static cudaError_t launch(const void *f, dim3 g, dim3 b, size_t smem)
{
    note("launch %s %u %u %u %u %zu\n", name_of(f), g.x, g.y, g.z, b.x * b.y * b.z, smem);
    return cudaSuccess;
}

/* what nvcc's host code calls */
void **__cudaRegisterFatBinary(void *bin)
{
    static void *handle;
    (void)bin;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterVar(void **h, char *v, char *a, const char *n, int e, size_t s, int c, int g)
{
    (void)h, (void)v, (void)a, (void)n, (void)e, (void)s, (void)c, (void)g;
}
void __cudaRegisterFunction(void **h, const char *host, char *dev, const char *name, int lim, uint3 *t, uint3 *b,
                            dim3 *bd, dim3 *gd, int *ws)
{
    (void)h, (void)dev, (void)lim, (void)t, (void)b, (void)bd, (void)gd, (void)ws;
    if (n_kernels < MAX_KERNELS) {
        funcs[n_kernels] = host;
        names[n_kernels++] = name;
    }
}
static __thread struct {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
} config;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st *stream)
{
    config.grid = grid;
    config.block = block;
    config.smem = smem;
    config.stream = stream;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream)
{
    *grid = config.grid;
    *block = config.block;
    *smem = config.smem;
    *(cudaStream_t *)stream = config.stream;
    return cudaSuccess;
}

cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v)
{
    note("attr %s %d %d\n", name_of(f), (int)a, v);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **args, size_t smem, cudaStream_t st)
{
    (void)args, (void)st;
    return launch(f, g, b, smem);
}
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3 b, void **args, size_t smem, cudaStream_t st)
{
    (void)args, (void)st;
    return launch(f, g, b, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args)
{
    (void)args;
    return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes);
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int t, size_t s, unsigned fl)
{
    (void)f, (void)t, (void)s, (void)fl;
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int dev)
{
    (void)dev;
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 227 * 1024 : 1;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d)
{
    (void)d;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "error"; }
cudaError_t cudaGetDriverEntryPoint(const char *s, void **f, unsigned long long fl, enum cudaDriverEntryPointQueryResult *r)
{
    (void)s, (void)fl, (void)r;
    *f = NULL;
    return cudaErrorNotSupported;
}
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p)
{
    (void)a, (void)p;
    return cudaErrorInvalidValue;
}

/* memory: host memory, zeroed */
cudaError_t cudaMalloc(void **p, size_t n) { return (*p = calloc(1, n ? n : 1)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaMallocHost(void **p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned fl)
{
    (void)fl;
    return cudaMalloc(p, n);
}
cudaError_t cudaFree(void *p)
{
    free(p);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
/* the copies and memsets are not carried out: the tests hand in made-up addresses */
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st)
{
    (void)d, (void)s, (void)st;
    note("copy %zu %d\n", n, (int)k);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) { return cudaMemcpyAsync(d, s, n, k, 0); }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st)
{
    (void)d, (void)v, (void)n, (void)st;
    return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { return cudaMemsetAsync(d, v, n, 0); }

/* streams and events: nothing to wait for */
static cudaError_t dummy(void **p)
{
    static char object;
    *p = &object;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return dummy((void **)e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned fl)
{
    (void)fl;
    return dummy((void **)e);
}
cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    (void)e;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st)
{
    (void)e, (void)st;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    (void)e;
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b)
{
    (void)a, (void)b;
    *ms = 0.f;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *st, unsigned fl)
{
    (void)fl;
    return dummy((void **)st);
}
cudaError_t cudaStreamDestroy(cudaStream_t st)
{
    (void)st;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st)
{
    (void)st;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned fl)
{
    (void)st, (void)e, (void)fl;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
