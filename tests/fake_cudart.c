/* A CUDA runtime without a GPU, for tests of the host side: memory is the host's, kernels do nothing, copies
 * run at once but stay "pending" until a synchronisation that covers them, and the n-th call that can fail
 * does (fake_fail_at). fake_pending counts what a caller would find in flight. */
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

#undef cudaGetDeviceProperties

enum { kOps = 1 << 16, kStreams = 64, kEvents = 256 };
typedef struct { int stream; long seq; int kind; /* 0 work, 1 wait for (other, upto) */ int other; long upto; int done; } Op;
static Op ops[kOps];
static int num_ops, num_streams = 1, num_events = 1;
static long seqs[kStreams];
static struct { int stream; long seq; } events[kEvents];
static long fail_at, calls;
static cudaError_t last_error;

void fake_fail_at(long n) { fail_at = n; calls = 0; last_error = cudaSuccess; }
long fake_calls(void) { return calls; }
void fake_reset(void) {
  num_ops = 0;
  num_streams = num_events = 1;
}
int fake_pending(void) {
  int n = 0;
  for (int i = 0; i < num_ops; ++i) n += ops[i].kind == 0 && !ops[i].done;
  return n;
}

static int id(cudaStream_t s) { return (int)(size_t)s % kStreams; }
static cudaError_t fails(cudaError_t e) {
  if (++calls != fail_at) return cudaSuccess;
  last_error = e;
  return e;
}
static void put(int stream, int kind, int other, long upto) {
  if (num_ops < kOps) ops[num_ops++] = (Op){stream, ++seqs[stream], kind, other, upto, 0};
}
static void complete(int stream, long upto) {
  for (int i = 0; i < num_ops; ++i) {
    if (ops[i].done || ops[i].stream != stream || ops[i].seq > upto) continue;
    ops[i].done = 1;
    if (ops[i].kind == 1) complete(ops[i].other, ops[i].upto);
  }
}

cudaError_t cudaGetLastError(void) { cudaError_t e = last_error; last_error = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t e) { (void)e; return "fake error"; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { (void)d; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp *p, int d) {
  (void)d;
  memset(p, 0, sizeof *p);
  p->major = 10;
  p->minor = 3;
  p->multiProcessorCount = 4;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) { (void)a; (void)d; *v = 4; return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int *a, int *b) { *a = *b = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int d) { (void)d; *p = 0; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, enum cudaMemPoolAttr a, void *v) { (void)p; (void)a; (void)v; return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *a, size_t *b) { *a = *b = (size_t)1 << 38; return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) {
  const cudaError_t e = fails(cudaErrorMemoryAllocation);
  if (e == cudaSuccess) *p = calloc(1, n);
  return e;
}
cudaError_t cudaMallocHost(void **p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t s) { (void)s; return cudaMalloc(p, n); }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeAsync(void *p, cudaStream_t s) { (void)s; free(p); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p) { (void)p; memset(a, 0, sizeof *a); return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *s) { (void)p; (void)s; return cudaErrorUnknown; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  const cudaError_t e = fails(cudaErrorUnknown);
  (void)k;
  if (e != cudaSuccess) return e;
  memcpy(d, s, n);
  put(id(st), 0, 0, 0);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) { (void)k; memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
  const cudaError_t e = fails(cudaErrorUnknown);
  if (e != cudaSuccess) return e;
  memset(d, v, n);
  put(id(st), 0, 0, 0);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = (cudaStream_t)(size_t)num_streams++; return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned f, int p) { (void)p; return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { complete(id(s), seqs[id(s)]); return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus *c) { (void)s; *c = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) {
  const cudaError_t r = fails(cudaErrorUnknown);
  (void)f;
  if (r == cudaSuccess) put(id(s), 1, events[(size_t)e].stream, events[(size_t)e].seq);
  return r;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s; (void)m; return cudaErrorUnknown; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) { (void)s; (void)g; return cudaErrorUnknown; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long f) { (void)x; (void)g; (void)f; return cudaErrorUnknown; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) { (void)x; (void)s; return cudaErrorUnknown; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { (void)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g) { (void)g; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void)f; *e = (cudaEvent_t)(size_t)num_events++; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  const cudaError_t r = fails(cudaErrorUnknown);
  if (r != cudaSuccess) return r;
  events[(size_t)e].stream = id(s);
  events[(size_t)e].seq = seqs[id(s)];
  return cudaSuccess;
}
cudaError_t cudaEventRecordWithFlags(cudaEvent_t e, cudaStream_t s, unsigned f) { (void)f; return cudaEventRecord(e, s); }
cudaError_t cudaEventQuery(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { complete(events[(size_t)e].stream, events[(size_t)e].seq); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t a, cudaEvent_t b) { (void)a; (void)b; *t = 0.0f; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) { (void)f; (void)a; (void)v; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int t, size_t b, unsigned g) { (void)f; (void)t; (void)b; (void)g; *n = 1; return cudaSuccess; }

/* What nvcc's host code calls to register and launch kernels. */
static cudaStream_t launch_stream;
void **__cudaRegisterFatBinary(void *b) { (void)b; static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterFunction(void **h, const char *f, char *n, const char *d, int l, void *t, void *b, void *g, void *w, int *s) {
  (void)h; (void)f; (void)n; (void)d; (void)l; (void)t; (void)b; (void)g; (void)w; (void)s;
}
void __cudaRegisterVar(void **h, char *v, char *a, const char *n, int e, size_t s, int c, int g) {
  (void)h; (void)v; (void)a; (void)n; (void)e; (void)s; (void)c; (void)g;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, cudaStream_t s) { (void)g; (void)b; (void)m; launch_stream = s; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *m, void *s) {
  g->x = g->y = g->z = b->x = b->y = b->z = 1;
  *m = 0;
  *(cudaStream_t *)s = launch_stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) { *k = (cudaKernel_t)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void **a, size_t m, cudaStream_t s) {
  const cudaError_t e = fails(cudaErrorUnknown);
  (void)k; (void)g; (void)b; (void)a; (void)m;
  if (e == cudaSuccess) put(id(s), 0, 0, 0);
  return e;
}
