/* A stand-in for the CUDA runtime on machines without a GPU (LD_PRELOAD): nothing runs, every kernel launch and every function
 * attribute is reported to a callback, whose return value becomes the call's result and, as in the real runtime, the calling
 * thread's pending error.  Device addresses are made up and never dereferenced. */
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <string.h>

static __thread cudaError_t g_pending = cudaSuccess;
static __thread struct { dim3 grid, block; size_t smem; cudaStream_t stream; } g_config;
static struct { const void* fn; const char* name; } g_kernels[256];
static int g_n_kernels;
static size_t g_next = (size_t)1 << 40;

typedef int (*launch_cb)(const char* name, unsigned grid, unsigned block, size_t smem, int cluster, int early, void** args);
typedef int (*call_cb)(const char* name, int value);
static launch_cb g_on_launch;
static call_cb g_on_smem_limit, g_on_call;
void fake_callbacks(launch_cb on_launch, call_cb on_smem_limit, call_cb on_call) { g_on_launch = on_launch; g_on_smem_limit = on_smem_limit; g_on_call = on_call; }
int fake_pending(void) { return g_pending; }

static cudaError_t result(int e) { if (e) g_pending = (cudaError_t)e; return (cudaError_t)e; }
static cudaError_t call(const char* name, size_t value) { return result(g_on_call ? g_on_call(name, (int)value) : 0); }
static const char* kernel_name(const void* fn) {
    for (int i = 0; i < g_n_kernels; ++i) if (g_kernels[i].fn == fn) return g_kernels[i].name;
    return "?";
}

void** __cudaRegisterFatBinary(void* p) { static void* handle[1]; (void)p; return handle; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterVar(void** h, char* v, char* a, const char* n, int e, size_t s, int c, int g) { (void)h; (void)v; (void)a; (void)n; (void)e; (void)s; (void)c; (void)g; }
void __cudaRegisterFunction(void** h, const char* fn, char* dev, const char* name, int t, void* a, void* b, void* c, void* d, int* w) {
    (void)h; (void)dev; (void)t; (void)a; (void)b; (void)c; (void)d; (void)w;
    if (g_n_kernels < 256) { g_kernels[g_n_kernels].fn = fn; g_kernels[g_n_kernels++].name = name; }
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st* s) {
    g_config.grid = g; g_config.block = b; g_config.smem = smem; g_config.stream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
    *g = g_config.grid; *b = g_config.block; *smem = g_config.smem; *(cudaStream_t*)s = g_config.stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* fn, dim3 g, dim3 b, void** args, size_t smem, cudaStream_t s) {
    (void)s;
    return result(g_on_launch ? g_on_launch(kernel_name(fn), g.x, b.x, smem, 0, 0, args) : 0);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void** args) {
    int cluster = 0, early = 0;
    for (unsigned i = 0; i < c->numAttrs; ++i) {
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cluster = (int)c->attrs[i].val.clusterDim.x;
        if (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization) early = c->attrs[i].val.programmaticStreamSerializationAllowed;
    }
    return result(g_on_launch ? g_on_launch(kernel_name(fn), c->gridDim.x, c->blockDim.x, c->dynamicSmemBytes, cluster, early, args) : 0);
}
cudaError_t cudaFuncSetAttribute(const void* fn, enum cudaFuncAttribute a, int v) {
    return result(a == cudaFuncAttributeMaxDynamicSharedMemorySize && g_on_smem_limit ? g_on_smem_limit(kernel_name(fn), v) : 0);
}
static CUresult encode(void* map) { memset(map, 0, sizeof(CUtensorMap)); return CUDA_SUCCESS; }
cudaError_t cudaGetDriverEntryPoint(const char* n, void** f, unsigned long long flags, enum cudaDriverEntryPointQueryResult* q) {
    (void)n; (void)flags;
    *f = (void*)encode;
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { cudaError_t e = g_pending; g_pending = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t e) { (void)e; return "made-up error"; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { (void)d; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) { (void)d; *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { cudaError_t e = call("cudaMalloc", n >> 20); *p = (void*)g_next; g_next += (n + 1023) & ~(size_t)1023; return e; }
cudaError_t cudaFree(void* p) { (void)p; return call("cudaFree", 0); }
cudaError_t cudaMemset(void* p, int v, size_t n) { (void)p; (void)v; return call("cudaMemset", n); }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) { (void)p; (void)v; (void)s; return call("cudaMemsetAsync", n); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) { (void)d; (void)s; (void)k; (void)st; return call("cudaMemcpyAsync", n); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return call("cudaStreamSynchronize", 0); }
cudaError_t cudaGetSymbolAddress(void** p, const void* sym) { (void)sym; *p = (void*)g_next; g_next += 16 << 20; return cudaSuccess; }
