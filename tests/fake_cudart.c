/* A stand-in for the CUDA runtime calls of libbcgpu.so (preloaded by
 * tests/test_failed_calls.py; no GPU): memory is host memory, copies and
 * kernels do nothing but stay "in flight" on their stream until the stream or
 * an event behind them is waited for, and the n-th call of a kind can be made
 * to fail.  fake_pending() counts what is still in flight. */
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

enum { LAUNCH, COPY, HOSTALLOC, KINDS };
static int fail_at[KINDS] = {-1, -1, -1}, calls[KINDS];
void fake_fail(int kind, int nth) {
  for (int k = 0; k < KINDS; k++) { fail_at[k] = -1; calls[k] = 0; }
  if (kind >= 0) fail_at[kind] = nth;
}
int fake_calls(int kind) { return calls[kind]; }
static cudaError_t last_error;
static int fails(int kind) {
  if (calls[kind]++ != fail_at[kind]) return 0;
  last_error = cudaErrorUnknown;
  return 1;
}
cudaError_t cudaGetLastError(void) {
  cudaError_t e = last_error;
  last_error = cudaSuccess;
  return e;
}

/* ---- operations in flight */
typedef struct { int prev, dep, done, work; } Op;
static Op ops[1 << 16];
static int nops;
struct CUstream_st { int last; };
struct CUevent_st { int op; };
static struct CUstream_st legacy = {-1};
static struct CUstream_st *st_of(cudaStream_t s) { return s ? s : &legacy; }
static void push(cudaStream_t s, int dep, int work) {
  if (nops == 1 << 16) abort();
  ops[nops] = (Op){st_of(s)->last, dep, 0, work};
  st_of(s)->last = nops++;
}
static void complete(int i) {
  for (; i >= 0 && !ops[i].done; i = ops[i].prev) {
    ops[i].done = 1;
    complete(ops[i].dep);
  }
}
int fake_pending(void) {
  int n = 0;
  for (int i = 0; i < nops; i++) n += ops[i].work && !ops[i].done;
  return n;
}
static cudaError_t work(cudaStream_t s, int kind) {
  if (fails(kind)) return cudaErrorUnknown;
  push(s, -1, 1);
  return cudaSuccess;
}

/* ---- memory: what is device and what is pinned memory */
static struct { char *p; size_t n; int type; } mem[4096];
static int nmem;
static cudaError_t take(void **p, size_t n, int type) {
  *p = malloc(n);
  if (nmem < 4096) { mem[nmem].p = *p; mem[nmem].n = n; mem[nmem++].type = type; }
  return cudaSuccess;
}
static cudaError_t give(void *p) {
  for (int i = 0; i < nmem; i++)
    if (mem[i].p == p) mem[i] = mem[--nmem];
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { return take(p, n, cudaMemoryTypeDevice); }
cudaError_t cudaFree(void *p) { return give(p); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t s) { return take(p, n, cudaMemoryTypeDevice); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t s) { return give(p); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned f) {
  return fails(HOSTALLOC) ? cudaErrorUnknown : take(p, n, cudaMemoryTypeHost);
}
cudaError_t cudaFreeHost(void *p) { return give(p); }
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *q) {
  memset(a, 0, sizeof *a);
  a->type = cudaMemoryTypeUnregistered;
  for (int i = 0; i < nmem; i++)
    if ((char *)q >= mem[i].p && (char *)q < mem[i].p + mem[i].n) a->type = mem[i].type;
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = (size_t)180 << 30; return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int d) { *p = 0; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, enum cudaMemPoolAttr a, void *v) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t n) { return cudaSuccess; }

/* ---- copies, kernels */
cudaError_t cudaMemcpyAsync(void *d, const void *q, size_t n, enum cudaMemcpyKind k, cudaStream_t s) {
  return work(s, COPY);
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t s) { push(s, -1, 1); return cudaSuccess; }
static int last_grid, clusters = 16;
int fake_last_grid(void) { return last_grid; }
void fake_clusters(int n) { clusters = n; }
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **a, size_t m, cudaStream_t s) {
  last_grid = g.x;
  return work(s, LAUNCH);
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *f, const cudaLaunchConfig_t *c) {
  *n = clusters;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **a) { return work(c->stream, LAUNCH); }
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3 b, void **a, size_t m, cudaStream_t s) {
  return work(s, LAUNCH);
}
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *f, int t, size_t m) {
  *n = 1;
  return cudaSuccess;
}

/* a <<<>>> launch: its shape, then cudaLaunchKernel */
static struct { dim3 g, b; size_t m; cudaStream_t s; } cfg;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, struct CUstream_st *s) {
  cfg.g = g; cfg.b = b; cfg.m = m; cfg.s = s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *m, void *s) {
  *g = cfg.g; *b = cfg.b; *m = cfg.m; *(cudaStream_t *)s = cfg.s;
  return cudaSuccess;
}

/* ---- streams and events */
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) {
  *s = malloc(sizeof **s);
  (*s)->last = -1;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { complete(st_of(s)->last); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { push(s, e->op, 0); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) {
  *e = malloc(sizeof **e);
  (*e)->op = -1;
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { e->op = st_of(s)->last; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { complete(e->op); return cudaSuccess; }
static int spans;
int fake_spans(void) { int n = spans; spans = 0; return n; } /* since the last call */
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) { spans++; *ms = 0; return cudaSuccess; }

/* ---- device */
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp *p, int d) {
  memset(p, 0, sizeof *p);
  p->major = 10;
  p->multiProcessorCount = 148;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *v) { return take(p, 16 << 20, cudaMemoryTypeDevice); }
const char *cudaGetErrorString(cudaError_t e) { return "made by the test"; }
static int encode_tensor_map() { return 0; }
cudaError_t cudaGetDriverEntryPointByVersion(const char *n, void **f, unsigned v, unsigned long long fl,
                                             enum cudaDriverEntryPointQueryResult *q) {
  *f = (void *)encode_tensor_map;
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

/* ---- the compiler's registration of kernels and variables */
void **__cudaRegisterFatBinary(void *b) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **h) {}
void __cudaUnregisterFatBinary(void **h) {}
void __cudaRegisterFunction(void **h, const char *f, char *d, const char *n, int t, void *a, void *b, void *c, void *e,
                            int *w) {}
void __cudaRegisterVar(void **h, char *v, char *a, const char *n, int e, size_t s, int c, int g) {}
