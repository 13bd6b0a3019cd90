/* A CUDA runtime without a GPU, preloaded over the real one by
 * test_pattern_failure.py and test_solve_failure.py: device memory is host
 * memory, kernels do nothing, the n-th allocation (device, pinned, event) fails
 * on request, the first 4-byte reads from the device return scripted values, a
 * read of the length of the row pointers returns rows of equal lengths, and reads
 * into pinned memory or of two doubles (a kernel's outcome) return ones. */
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

static size_t g_live;         /* bytes of device memory */
static char* g_pinned;        /* the last pinned allocation */
static size_t g_pinned_size;
static int g_mallocs, g_fail_at = -1, g_script[8], g_reads, g_edge_passes, g_null_edge_lists;

/* Allocations are counted from 0 here; fail_at < 0: none fails. */
void fake_reset(int fail_at, int read0, int read1) {
    g_mallocs = g_reads = g_edge_passes = g_null_edge_lists = 0;
    g_fail_at = fail_at;
    g_script[0] = read0;
    g_script[1] = read1;
}
static int g_rows, g_per_row;
void fake_rows(int rows, int per_row) {
    g_rows = rows;
    g_per_row = per_row;
}
int fake_mallocs(void) { return g_mallocs; }
size_t fake_live(void) { return g_live; }
int fake_edge_passes(void) { return g_edge_passes; }
int fake_null_edge_lists(void) { return g_null_edge_lists; }

static int refused(void) { return g_mallocs++ == g_fail_at; }
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = NULL;
    if (refused()) return cudaErrorMemoryAllocation;
    size_t* q = calloc(256 + n, 1);   /* the size, then memory aligned as malloc aligns */
    if (!q) return cudaErrorMemoryAllocation;
    *q = n;
    g_live += n;
    *p = (char*)q + 256;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (!p) return cudaSuccess;
    size_t* q = (size_t*)((char*)p - 256);
    g_live -= *q;
    free(q);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned flags) {
    (void)flags;
    *p = NULL;
    if (refused()) return cudaErrorMemoryAllocation;
    *p = g_pinned = calloc(n, 1);
    g_pinned_size = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    if (p == g_pinned) g_pinned_size = 0;
    free(p);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    if (refused()) return cudaErrorMemoryAllocation;
    *e = (cudaEvent_t)1;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) { (void)st; return e ? cudaSuccess : cudaErrorInvalidValue; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
    *ms = 1.f;
    return a && b ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind kind, cudaStream_t st) {
    (void)st;
    if (n && (!d || !s)) return cudaErrorInvalidValue;
    if (kind == cudaMemcpyDeviceToHost && n == 4 && g_reads < 2)
        *(int*)d = g_script[g_reads++];
    else if (kind == cudaMemcpyDeviceToHost && g_rows && n == 4 * ((size_t)g_rows + 1))
        for (int i = 0; i <= g_rows; ++i) ((int*)d)[i] = i * g_per_row;
    else if (kind == cudaMemcpyDeviceToHost &&
             (n == 16 || ((char*)d >= g_pinned && (char*)d < g_pinned + g_pinned_size)))
        for (size_t i = 0; i < n / sizeof(double); ++i) ((double*)d)[i] = 1.0;
    else
        memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbolAsync(const void* sym, const void* s, size_t n, size_t off, enum cudaMemcpyKind kind,
                                    cudaStream_t st) {
    (void)sym, (void)s, (void)n, (void)off, (void)kind, (void)st;
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
    if (n && !d) return cudaErrorInvalidValue;
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) { (void)st; return cudaMemset(d, v, n); }

/* Kernels by name: the edge pass must get its list of slots. */
static const void* g_edge_kernel;
void** __cudaRegisterFatBinary(void* bin) { static void* h; (void)bin; return &h; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterVar(void** h, char* a, char* b, const char* c, int d, size_t e, int f, int g) {
    (void)h, (void)a, (void)b, (void)c, (void)d, (void)e, (void)f, (void)g;
}
void __cudaRegisterFunction(void** h, const char* host, char* dev, const char* name, int lim, void* a, void* b, void* c,
                            void* d, int* e) {
    (void)h, (void)dev, (void)lim, (void)a, (void)b, (void)c, (void)d, (void)e;
    if (strstr(name, "k_edge_pass")) g_edge_kernel = host;
}
static struct {
    dim3 grid, block;
    size_t smem;
    void* stream;
} g_cfg;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void* stream) {
    g_cfg.grid = grid;
    g_cfg.block = block;
    g_cfg.smem = smem;
    g_cfg.stream = stream;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
    *grid = g_cfg.grid;
    *block = g_cfg.block;
    *smem = g_cfg.smem;
    *(void**)stream = g_cfg.stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t st) {
    (void)grid, (void)block, (void)smem, (void)st;
    if (f == g_edge_kernel) {
        ++g_edge_passes;
        if (*(void**)args[0] == NULL) ++g_null_edge_lists;
    }
    return cudaSuccess;
}
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t st) {
    return cudaLaunchKernel(f, grid, block, args, smem, st);
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
    (void)f, (void)a, (void)v;
    return cudaSuccess;
}

cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int dev) {
    (void)dev;
    *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrComputeCapabilityMinor ? 0 : 148;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void* f) {
    (void)f;
    memset(a, 0, sizeof(*a));
    a->ptxVersion = a->binaryVersion = 100;
    a->maxThreadsPerBlock = 1024;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int block, size_t smem,
                                                                   unsigned flags) {
    (void)f, (void)block, (void)smem, (void)flags;
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int block, size_t smem) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(n, f, block, smem, 0);
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { (void)d; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaPeekAtLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned flags) { (void)flags; *s = (cudaStream_t)1; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
