/* A CUDA runtime without a GPU, for tests of the host code's stream order: memory is host memory, kernels do nothing, copies are
 * made at once, and every operation on a stream is counted.  Events carry what their stream was ordered after, so that
 * fake_unordered() can tell how many operations of other streams a stream (or the host) has not been made to wait for.
 * fake_fail_at(n) lets the n-th fallible call from then on return cudaErrorMemoryAllocation.  A capture records nothing, its
 * operations count like others; it ends with an error while a stream is not joined.  Memory is zero at first (from 32 MB on it comes
 * from the system).  fake_graph_flags(): of the last instantiation. */
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

enum { MAX_STREAMS = 64 };
typedef struct { unsigned long long at[MAX_STREAMS]; } Clock;
struct CUstream_st { int id; };
struct CUevent_st { Clock c; };
static struct CUstream_st streams[MAX_STREAMS];
static int n_streams = 1;                               /* 0: the default stream */
static unsigned long long done[MAX_STREAMS];            /* operations enqueued so far */
static Clock known[MAX_STREAMS], host;
static long calls, fail_at = -1, waits;
static dim3 cfg_grid, cfg_block;
static size_t cfg_smem;
static cudaStream_t cfg_stream;
static long graph_flags = -1;

static int id_of(cudaStream_t s) { return s ? s->id : 0; }
static void op(cudaStream_t s) { int i = id_of(s); known[i].at[i] = ++done[i]; }
static void merge(Clock* a, const Clock* b) { for (int i = 0; i < MAX_STREAMS; i++) if (b->at[i] > a->at[i]) a->at[i] = b->at[i]; }
static cudaError_t last_error;                          /* of this thread's calls, until it is asked for */
static cudaError_t fallible(void) { return calls++ == fail_at ? (last_error = cudaErrorMemoryAllocation) : cudaSuccess; }
#define FALLIBLE do { cudaError_t e_ = fallible(); if (e_) return e_; } while (0)

long fake_calls(void) { return calls; }
long fake_waits(void) { return waits; }                 /* of the host for a stream */
long fake_graph_flags(void) { return graph_flags; }
void fake_fail_at(long n) { calls = 0; fail_at = n; }
long fake_unordered(cudaStream_t s) {
    long n = 0;
    for (int i = 0; i < n_streams; i++) {
        const unsigned long long k = known[id_of(s)].at[i] > host.at[i] ? known[id_of(s)].at[i] : host.at[i];
        if (i != id_of(s)) n += (long)(done[i] - k);
    }
    return n;
}

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { (void)d; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(struct cudaDeviceProp* p, int d) { (void)d; memset(p, 0, sizeof *p); p->major = 10; p->multiProcessorCount = 148; return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) { *lo = 0; *hi = -5; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e ? "planted by the fake runtime" : "no error"; }
cudaError_t cudaGetLastError(void) { cudaError_t e = last_error; last_error = cudaSuccess; return e; }
cudaError_t cudaMalloc(void** p, size_t n) { FALLIBLE; *p = NULL; void* q = NULL; if (posix_memalign(&q, 256, n ? n : 1)) return cudaErrorMemoryAllocation; if (n < (32u << 20)) memset(q, 0, n); *p = q; return cudaSuccess; }
cudaError_t cudaFree(void* p) { for (int i = 0; i < n_streams; i++) host.at[i] = done[i]; free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned f) { (void)f; FALLIBLE; *p = calloc(n ? n : 1, 1); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) { (void)k; memmove(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyToSymbol(const void* y, const void* s, size_t n, size_t o, enum cudaMemcpyKind k) { (void)y; (void)s; (void)n; (void)o; (void)k; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) { (void)k; FALLIBLE; memmove(d, s, n); op(st); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) { FALLIBLE; memset(d, v, n); op(st); return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) { (void)f; (void)a; (void)v; FALLIBLE; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) { (void)f; FALLIBLE; streams[n_streams].id = n_streams; *s = &streams[n_streams++]; return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int p) { (void)p; return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { waits++; merge(&host, &known[id_of(s)]); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)f; FALLIBLE; merge(&known[id_of(s)], &e->c); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { FALLIBLE; *e = calloc(1, sizeof **e); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) { (void)f; return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { FALLIBLE; e->c = known[id_of(s)]; return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, struct CUstream_st* s) { cfg_grid = g; cfg_block = b; cfg_smem = m; cfg_stream = s; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) { *g = cfg_grid; *b = cfg_block; *m = cfg_smem; *(cudaStream_t*)s = cfg_stream; return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** a, size_t m, cudaStream_t s) { (void)f; (void)g; (void)b; (void)a; (void)m; op(s); return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a) { (void)f; (void)a; FALLIBLE; op(c->stream); return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s; (void)m; FALLIBLE; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
    FALLIBLE;
    *g = fake_unordered(s) ? NULL : (cudaGraph_t)&graph_flags;
    return *g ? cudaSuccess : cudaErrorStreamCaptureUnjoined;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long f) { FALLIBLE; *e = (cudaGraphExec_t)g; graph_flags = (long)f; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) { (void)e; FALLIBLE; op(s); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { (void)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { (void)e; return cudaSuccess; }
void** __cudaRegisterFatBinary(void* f) { static void* h; (void)f; return &h; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterFunction(void** h, const char* a, char* b, const char* c, int d, void* e, void* f, void* g, void* i, int* j) { (void)h; (void)a; (void)b; (void)c; (void)d; (void)e; (void)f; (void)g; (void)i; (void)j; }
void __cudaRegisterVar(void** h, char* a, char* b, const char* c, int d, size_t e, int f, int g) { (void)h; (void)a; (void)b; (void)c; (void)d; (void)e; (void)f; (void)g; }
