/* A CUDA runtime without a GPU, preloaded in front of libcudart for tests of the
 * library's host side: device memory is host memory, copies are memcpy, kernels are
 * counted and not run.  A launch on a stream of another device than the current one
 * fails, as on a GPU. */
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

#define MAX_KERNELS 4096
#define MAX_BLOCKS 4096

static _Thread_local int current = 0;
static struct { const void* fn; const char* name; int launches; } kernels[MAX_KERNELS];
static int n_kernels = 0;
static struct { char* p; size_t n; int dev; } blocks[MAX_BLOCKS];
static long long live = 0;                 /* bytes allocated and not freed */
static long long limit = 1LL << 60;        /* bytes there are */
static int capturing = 0;
static const float* elapsed = 0;           /* what the next event pairs measure */
static int n_elapsed = 0;
struct CUstream_st { int dev; };
struct CUevent_st { int dev; };

/* what a test reads and sets */
long long fake_live_bytes(void) { return live; }
void fake_capture(int on) { capturing = on; }   /* of a stream that is not the library's, waiting forbidden */
void fake_memory(long long bytes) { limit = bytes; }
int fake_launches(const char* part) {      /* launches of kernels whose name holds part */
  int s = 0;
  for (int k = 0; k < n_kernels; ++k)
    if (strstr(kernels[k].name, part)) s += kernels[k].launches;
  return s;
}
int fake_most_launches(void) {             /* of any one stage kernel */
  int s = 0;
  for (int k = 0; k < n_kernels; ++k)
    if (strstr(kernels[k].name, "stage_kernel") && kernels[k].launches > s) s = kernels[k].launches;
  return s;
}
void fake_reset(void) { for (int k = 0; k < n_kernels; ++k) kernels[k].launches = 0; }
void fake_elapsed(const float* ms, int n) { elapsed = ms; n_elapsed = n; }

/* the library's kernels */
void** __cudaRegisterFatBinary(void* b) { static void* h; (void)b; return &h; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterVar(void** h, char* v, char* d, const char* n, int e, size_t s, int c, int g) {
  (void)h; (void)v; (void)d; (void)n; (void)e; (void)s; (void)c; (void)g;
}
void __cudaRegisterFunction(void** h, const char* fn, char* d, const char* name, int t, void* ti, void* bi, void* bd,
                            void* gd, int* w) {
  (void)h; (void)d; (void)t; (void)ti; (void)bi; (void)bd; (void)gd; (void)w;
  if (n_kernels < MAX_KERNELS) { kernels[n_kernels].fn = fn; kernels[n_kernels++].name = name; }
}
static struct { dim3 g, b; size_t smem; void* st; } cfg;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* st) {
  cfg.g = g; cfg.b = b; cfg.smem = smem; cfg.st = st;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
  *g = cfg.g; *b = cfg.b; *smem = cfg.smem; *(void**)st = cfg.st;
  return cudaSuccess;
}
static cudaError_t launch(const void* fn, cudaStream_t st) {
  if (st && st->dev != current) return cudaErrorInvalidResourceHandle;
  for (int k = 0; k < n_kernels; ++k)
    if (kernels[k].fn == fn) { ++kernels[k].launches; return cudaSuccess; }
  return cudaErrorInvalidDeviceFunction;
}
cudaError_t cudaLaunchKernel(const void* fn, dim3 g, dim3 b, void** a, size_t s, cudaStream_t st) {
  (void)g; (void)b; (void)a; (void)s;
  return launch(fn, st);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void** a) { (void)a; return launch(fn, c->stream); }
cudaError_t cudaFuncSetAttribute(const void* fn, enum cudaFuncAttribute a, int v) { (void)fn; (void)a; (void)v; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* fn, int t, size_t s) {
  (void)fn; (void)t; (void)s;
  *n = 2;
  return cudaSuccess;
}

/* devices */
cudaError_t cudaGetDeviceCount(int* n) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { if (d < 0 || d > 1) return cudaErrorInvalidDevice; current = d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) { (void)a; (void)d; *v = 148; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char* n, void** f, unsigned v, unsigned long long fl,
                                             enum cudaDriverEntryPointQueryResult* q) {
  (void)n; (void)v; (void)fl;
  *f = 0;
  *q = cudaDriverEntryPointSymbolNotFound;
  return cudaSuccess;
}

/* memory */
cudaError_t cudaMalloc(void** p, size_t n) {
  if (live + (long long)n > limit) return cudaErrorMemoryAllocation;
  for (int k = 0; k < MAX_BLOCKS; ++k)
    if (!blocks[k].p) {
      if (!(*p = calloc(n ? n : 1, 1))) return cudaErrorMemoryAllocation;
      blocks[k].p = *p; blocks[k].n = n; blocks[k].dev = current;
      live += (long long)n;
      return cudaSuccess;
    }
  return cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void* p) {
  for (int k = 0; p && k < MAX_BLOCKS; ++k)
    if (blocks[k].p == p) { live -= (long long)blocks[k].n; blocks[k].p = 0; free(p); }
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes* a, const void* p) {
  memset(a, 0, sizeof *a);
  for (int k = 0; k < MAX_BLOCKS; ++k)
    if (blocks[k].p && (const char*)p >= blocks[k].p && (const char*)p < blocks[k].p + blocks[k].n) {
      a->type = cudaMemoryTypeDevice;
      a->device = blocks[k].dev;
    }
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { (void)s; *p = 0; return cudaErrorInvalidSymbol; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  (void)k; (void)st;
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, enum cudaMemcpyKind k,
                              cudaStream_t st) {
  (void)k; (void)st;
  for (size_t j = 0; j < h; ++j) memcpy((char*)d + j * dp, (const char*)s + j * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) { (void)st; memset(d, v, n); return cudaSuccess; }

/* streams, events, graphs */
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) {
  (void)f;
  *s = malloc(sizeof **s);
  (*s)->dev = current;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return capturing ? cudaErrorStreamCaptureUnsupported : cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t s) { (void)s; return capturing ? cudaErrorStreamCaptureUnsupported : cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s; (void)e; (void)f; return cudaSuccess; }
cudaError_t cudaStreamGetDevice(cudaStream_t s, int* d) { *d = s->dev; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus* c) {
  (void)s;
  *c = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s; (void)m; return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) { (void)s; *g = 0; return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { (void)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g) { (void)g; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long f) {
  (void)g; (void)f;
  *e = 0;
  return cudaErrorNotSupported;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t g, cudaStream_t s) { (void)g; (void)s; return cudaErrorNotSupported; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = malloc(sizeof **e); (*e)->dev = current; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) { (void)f; return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
  (void)a; (void)b;
  *ms = n_elapsed > 0 ? (--n_elapsed, *elapsed++) : 1.0f;
  return cudaSuccess;
}
