/* A stand-in for the CUDA runtime, preloaded before the library, so that the
 * host side of a match runs without a GPU: device memory is host memory,
 * kernels are logged and not run, and an allocation can be made to fail. */
#include <cuda_runtime_api.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

typedef struct { const void* fun; char name[64]; } Kernel;
static Kernel kernels[64];
static int nkernels;
typedef struct { void* p; size_t n; } Block;
static Block blocks[4096];
static int nblocks;

/* what a test reads and sets */
char fake_log[1 << 20];        /* "kernel grid block;" per launch, "copy bytes;" per asynchronous copy */
size_t fake_fail_at;           /* an allocation of at least this many bytes fails (0: none) */
size_t fake_fail_below;        /* and below this many (0: no upper limit) */
long fake_live, fake_instantiated;
static size_t at;
static int capturing;

void fake_reset(void) { at = 0; fake_log[0] = 0; }
static void put(const char* what, unsigned long a, unsigned long b) {
  if (at + 128 < sizeof(fake_log)) at += (size_t)sprintf(fake_log + at, "%s %lu %lu;", what, a, b);
}

void** __cudaRegisterFatBinary(void* f) { (void)f; static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterVar(void** h, char* a, char* b, const char* c, int d, size_t e, int f, int g) {
  (void)h, (void)a, (void)b, (void)c, (void)d, (void)e, (void)f, (void)g;
}
void __cudaRegisterFunction(void** h, const char* fun, char* dev, const char* name, int limit, uint3* t, uint3* b,
                            dim3* bd, dim3* gd, int* w) {
  (void)h, (void)dev, (void)limit, (void)t, (void)b, (void)bd, (void)gd, (void)w;
  if (nkernels == 64) abort();
  kernels[nkernels].fun = fun;
  snprintf(kernels[nkernels++].name, 64, "%s", name);
}
static dim3 cfg_grid, cfg_block;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, void* st) {
  (void)s, (void)st;
  cfg_grid = g, cfg_block = b;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) {
  *g = cfg_grid, *b = cfg_block, *s = 0;
  *(void**)st = NULL;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** args, size_t s, cudaStream_t st) {
  (void)args, (void)s, (void)st;
  for (int i = 0; i < nkernels; i++)
    if (kernels[i].fun == f) put(kernels[i].name, g.x, b.x);
  return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t n) {
  *p = NULL;
  if (fake_fail_at && n >= fake_fail_at && (!fake_fail_below || n < fake_fail_below)) return cudaErrorMemoryAllocation;
  *p = aligned_alloc(256, (n + 511) / 256 * 256);
  if (nblocks == 4096) abort();
  blocks[nblocks].p = *p;
  blocks[nblocks++].n = n;
  fake_live += (long)n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (!p) return cudaSuccess;
  for (int i = 0; i < nblocks; i++)
    if (blocks[i].p == p) {
      fake_live -= (long)blocks[i].n;
      blocks[i] = blocks[--nblocks];
      free(p);
      return cudaSuccess;
    }
  fprintf(stderr, "freed twice or not device memory\n");
  abort();
}
static void owned(const void* p, size_t n) {  /* a copy or memset of device memory stays inside it */
  for (int i = 0; i < nblocks; i++)
    if ((const char*)p >= (char*)blocks[i].p && (const char*)p + n <= (char*)blocks[i].p + blocks[i].n) return;
  fprintf(stderr, "%zu bytes outside device memory\n", n);
  abort();
}
cudaError_t cudaMallocHost(void** p, size_t n) { *p = calloc(1, n ? n : 1); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned f) { (void)f; return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) {
  if (k != cudaMemcpyDeviceToHost) owned(d, n);
  if (k != cudaMemcpyHostToDevice) owned(s, n);
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  (void)st;
  put("copy", n, 0);
  return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void* p, int v, size_t n) { owned(p, n); memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) { (void)st; return cudaMemset(p, v, n); }

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return d == 0 ? cudaSuccess : cudaErrorInvalidDevice; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) { (void)a, (void)d; *v = 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) { (void)f, (void)a, (void)v; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int b, size_t s, unsigned fl) {
  (void)f, (void)b, (void)s, (void)fl;
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes* a, const void* p) {
  memset(a, 0, sizeof(*a));
  a->type = cudaMemoryTypeUnregistered;
  a->device = -1;
  for (int i = 0; i < nblocks; i++)
    if ((const char*)p >= (char*)blocks[i].p && (const char*)p < (char*)blocks[i].p + blocks[i].n) {
      a->type = cudaMemoryTypeDevice;
      a->device = 0;
    }
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char* s, void** f, unsigned long long fl, enum cudaDriverEntryPointQueryResult* q) {
  (void)s, (void)fl;
  *f = NULL;
  *q = cudaDriverEntryPointSymbolNotFound;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { (void)s; *p = NULL; return cudaErrorInvalidSymbol; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorName(cudaError_t e) { (void)e; return "error"; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }

static int object;
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)&object; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) { (void)f; return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t a, cudaEvent_t b) { (void)a, (void)b; *t = 0; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e, (void)s; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) { (void)f; *s = (cudaStream_t)&object; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s, (void)e, (void)f; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus* c) {
  *c = s && capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s, (void)m; capturing = 1; return cudaSuccess; }
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t s, cudaGraph_t g, const cudaGraphNode_t* d, const cudaGraphEdgeData* e,
                                          size_t n, enum cudaStreamCaptureMode m) {
  (void)s, (void)g, (void)d, (void)e, (void)n, (void)m;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) { (void)s; capturing = 0; *g = (cudaGraph_t)&object; return cudaSuccess; }
cudaError_t cudaGraphCreate(cudaGraph_t* g, unsigned f) { (void)f; *g = (cudaGraph_t)&object; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { (void)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g) { (void)g; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long f) {
  (void)g, (void)f;
  *e = (cudaGraphExec_t)&object;
  fake_instantiated++;
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) { (void)e, (void)s; put("graph", 0, 0); return cudaSuccess; }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle* h, cudaGraph_t g, unsigned d, unsigned f) {
  (void)g, (void)d, (void)f;
  *h = 1;
  return cudaSuccess;
}
cudaError_t cudaGraphAddKernelNode(cudaGraphNode_t* n, cudaGraph_t g, const cudaGraphNode_t* d, size_t k, const struct cudaKernelNodeParams* p) {
  (void)g, (void)d, (void)k, (void)p;
  *n = (cudaGraphNode_t)&object;
  return cudaSuccess;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t* n, cudaGraph_t g, const cudaGraphNode_t* d, size_t k, struct cudaGraphNodeParams* p) {
  static cudaGraph_t body = (cudaGraph_t)&object;
  (void)g, (void)d, (void)k;
  *n = (cudaGraphNode_t)&object;
  p->conditional.phGraph_out = &body;
  return cudaSuccess;
}
