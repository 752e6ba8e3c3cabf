/* A CUDA runtime without a GPU, for tests of the host code: the objects of
 * libmdforce are linked against it in place of cudart.  Memory is host memory,
 * copies are carried out, kernels are only looked at: their limits are checked
 * and their names logged.  Two devices.  fake_fail_at(k) makes the k-th call
 * from now on that can fail return an error, as the real one would. */
#include <cuda_runtime_api.h>
#include <pthread.h>
#include <stdlib.h>
#include <string.h>

#define DEVICES 2
#define MAX_BLOCKS 65536
#define MAX_FUNCS 4096
#define MAX_LOG 65536

enum { DEVICE_MEM, POOL_MEM, PINNED_MEM };

static struct { char* p; size_t bytes; int kind; } blocks[MAX_BLOCKS];
static struct { const void* f; const char* name; int limit[DEVICES], used[DEVICES], lowered; } funcs[MAX_FUNCS];
static struct { int func, device; size_t smem; } launches[MAX_LOG];
static int nblocks, nfuncs, nlaunches, streams, trims;
static size_t pageable_dtoh;
static int unordered;
static long calls, fail_at = -1;
static pthread_mutex_t mutex = PTHREAD_MUTEX_INITIALIZER;
static __thread int device;
static __thread cudaError_t last;
static __thread struct { dim3 g, b; size_t smem; cudaStream_t s; } config;

static cudaError_t fail(cudaError_t e) { last = e; return e; }

/* counts one call that can fail; true: it fails */
static int fails(void) {
  pthread_mutex_lock(&mutex);
  const int hit = calls++ == fail_at;
  pthread_mutex_unlock(&mutex);
  return hit;
}
#define MAY_FAIL(e) if (fails()) return fail(e)

static cudaError_t take(void** p, size_t bytes, int kind) {
  char* q = calloc(1, bytes ? bytes : 1);
  pthread_mutex_lock(&mutex);
  int k = 0;
  while (k < nblocks && blocks[k].p) ++k;
  if (k == nblocks) ++nblocks;
  blocks[k].p = q;
  blocks[k].bytes = bytes;
  blocks[k].kind = kind;
  pthread_mutex_unlock(&mutex);
  *p = q;
  return cudaSuccess;
}

static cudaError_t drop(void* p) {
  pthread_mutex_lock(&mutex);
  for (int k = 0; p && k < nblocks; ++k)
    if (blocks[k].p == (char*)p) { free(p); blocks[k].p = NULL; p = NULL; }
  pthread_mutex_unlock(&mutex);
  return p ? fail(cudaErrorInvalidValue) : cudaSuccess;
}

static int pinned(const void* p) {
  for (int k = 0; k < nblocks; ++k)
    if (blocks[k].p && blocks[k].kind == PINNED_MEM && (char*)p >= blocks[k].p && (char*)p < blocks[k].p + blocks[k].bytes)
      return 1;
  return 0;
}

static int find(const void* f) {
  for (int k = 0; k < nfuncs; ++k)
    if (funcs[k].f == f) return k;
  return -1;
}

static cudaError_t launch(const void* f, dim3 g, dim3 b, size_t smem) {
  MAY_FAIL(cudaErrorLaunchOutOfResources);
  const int k = find(f);
  if (k < 0) return fail(cudaErrorInvalidDeviceFunction);
  if (!g.x || !g.y || !g.z || g.y > 65535 || g.z > 65535 || b.x * b.y * b.z > 1024 || !b.x || !b.y || !b.z)
    return fail(cudaErrorInvalidConfiguration);
  if (smem > (size_t)(funcs[k].limit[device] ? funcs[k].limit[device] : 48 * 1024)) return fail(cudaErrorInvalidValue);
  pthread_mutex_lock(&mutex);
  if ((int)smem > funcs[k].used[device]) funcs[k].used[device] = (int)smem;
  if (nlaunches < MAX_LOG) {
    launches[nlaunches].func = k;
    launches[nlaunches].device = device;
    launches[nlaunches++].smem = smem;
  }
  pthread_mutex_unlock(&mutex);
  return cudaSuccess;
}

/* ------------------------------------------------------------ for the test */
void fake_reset(void) { calls = 0; fail_at = -1; nlaunches = 0; pageable_dtoh = 0; last = cudaSuccess; device = 0; trims = 0; }
void fake_fail_at(long k) { calls = 0; fail_at = k; }
long fake_calls(void) { return calls; }
long fake_live(void) {  /* bytes held, page-locked memory apart, streams and events */
  long n = streams;
  for (int k = 0; k < nblocks; ++k)
    if (blocks[k].p && blocks[k].kind != PINNED_MEM) n += (long)blocks[k].bytes;
  return n;
}
long fake_pinned(void) {
  long n = 0;
  for (int k = 0; k < nblocks; ++k)
    if (blocks[k].p && blocks[k].kind == PINNED_MEM) n += (long)blocks[k].bytes;
  return n;
}
long fake_pageable_dtoh(void) { return (long)pageable_dtoh; }
int fake_trims(void) { return trims; }
int fake_unordered(void) { return unordered; }  /* writes to the device that no stream of the library waits for */
int fake_launches(void) { return nlaunches; }
const char* fake_launch_name(int k) { return funcs[launches[k].func].name; }
/* a kernel whose shared-memory limit was taken below what it has been launched with */
const char* fake_lowered(void) {
  for (int k = 0; k < nfuncs; ++k)
    if (funcs[k].lowered) return funcs[k].name;
  return NULL;
}
/* a kernel launched with dynamic shared memory on a device where its limit was not set, though it was on another */
const char* fake_unprepared(void) {
  for (int k = 0; k < nfuncs; ++k)
    for (int d = 0; d < DEVICES; ++d)
      if (funcs[k].used[d] && !funcs[k].limit[d] && funcs[k].limit[!d]) return funcs[k].name;
  return NULL;
}

/* ------------------------------------------------------------ the runtime */
void** __cudaRegisterFatBinary(void* b) { static void* h; (void)b; return &h; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterVar(void** h, char* v, char* a, const char* n, int e, size_t s, int c, int g) {
  (void)h; (void)v; (void)a; (void)n; (void)e; (void)s; (void)c; (void)g;
}
void __cudaRegisterFunction(void** h, const char* f, char* d, const char* name, int l, uint3* t, uint3* b, dim3* bd,
                            dim3* gd, int* w) {
  (void)h; (void)d; (void)l; (void)t; (void)b; (void)bd; (void)gd; (void)w;
  if (nfuncs == MAX_FUNCS) abort();
  funcs[nfuncs].f = f;
  funcs[nfuncs].name = name;
  ++nfuncs;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st* s) {
  config.g = g; config.b = b; config.smem = smem; config.s = s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = config.g; *b = config.b; *smem = config.smem; *(cudaStream_t*)s = config.s;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** a, size_t smem, cudaStream_t s) {
  (void)a; (void)s;
  return launch(f, g, b, smem);
}
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 g, dim3 b, void** a, size_t smem, cudaStream_t s) {
  (void)a; (void)s;
  return launch(f, g, b, smem);
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute attr, int v) {
  MAY_FAIL(cudaErrorInvalidValue);
  const int k = find(f);
  if (k < 0) return fail(cudaErrorInvalidDeviceFunction);
  if (attr == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    if (v > 227 * 1024) return fail(cudaErrorInvalidValue);
    if (v < funcs[k].used[device]) funcs[k].lowered = 1;
    funcs[k].limit[device] = v;
  }
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "an error"; }
cudaError_t cudaGetDeviceCount(int* n) { *n = DEVICES; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) {
  if (d < 0 || d >= DEVICES) return fail(cudaErrorInvalidDevice);
  device = d;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) {
  (void)d;
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrCooperativeLaunch ? 1 : 0;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int b, size_t smem) {
  (void)f; (void)b; (void)smem;
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { MAY_FAIL(cudaErrorMemoryAllocation); return take(p, n, DEVICE_MEM); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t s) {
  (void)s;
  MAY_FAIL(cudaErrorMemoryAllocation);
  return take(p, n, DEVICE_MEM);
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t s) {
  (void)pool; (void)s;
  MAY_FAIL(cudaErrorMemoryAllocation);
  return take(p, n, POOL_MEM);
}
cudaError_t cudaMallocHost(void** p, size_t n) { MAY_FAIL(cudaErrorMemoryAllocation); return take(p, n, PINNED_MEM); }
cudaError_t cudaFree(void* p) { return drop(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) { (void)s; return drop(p); }
cudaError_t cudaFreeHost(void* p) { return drop(p); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const struct cudaMemPoolProps* props) {
  (void)props;
  *p = (cudaMemPool_t)&trims;
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, enum cudaMemPoolAttr a, void* v) { (void)p; (void)a; (void)v; return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t n) { (void)p; (void)n; ++trims; return cudaSuccess; }
static void copied(void* d, const void* s, size_t n, enum cudaMemcpyKind k) {
  memcpy(d, s, n);
  if (k != cudaMemcpyDeviceToHost) return;
  pthread_mutex_lock(&mutex);
  if (!pinned(d)) pageable_dtoh += n;
  pthread_mutex_unlock(&mutex);
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) {
  MAY_FAIL(cudaErrorInvalidValue);
  copied(d, s, n, k);
  if (k == cudaMemcpyHostToDevice) ++unordered;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  (void)st;
  MAY_FAIL(cudaErrorInvalidValue);
  copied(d, s, n, k);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { MAY_FAIL(cudaErrorInvalidValue); memset(p, v, n); ++unordered; return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
  (void)s;
  MAY_FAIL(cudaErrorInvalidValue);
  memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) {
  static char handles[1 << 16];
  static int n;
  (void)f;
  MAY_FAIL(cudaErrorMemoryAllocation);
  pthread_mutex_lock(&mutex);
  ++streams;
  *s = (cudaStream_t)(handles + (n++ & 0xffff));
  pthread_mutex_unlock(&mutex);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  (void)s;
  pthread_mutex_lock(&mutex);
  --streams;
  pthread_mutex_unlock(&mutex);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; MAY_FAIL(cudaErrorUnknown); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) {
  (void)f;
  return cudaStreamCreateWithFlags((cudaStream_t*)e, 0);
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { return cudaStreamDestroy((cudaStream_t)e); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; MAY_FAIL(cudaErrorUnknown); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; MAY_FAIL(cudaErrorUnknown); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes* a, const void* p) {
  (void)p;
  memset(a, 0, sizeof(*a));
  a->type = cudaMemoryTypeDevice;
  return cudaSuccess;
}
/* graphs, mapped host memory and symbols: not part of these tests */
#define NONE(name, args) cudaError_t name args { return fail(cudaErrorNotSupported); }
NONE(cudaHostRegister, (void* p, size_t n, unsigned f))
NONE(cudaHostUnregister, (void* p))
NONE(cudaHostGetDevicePointer, (void** d, void* p, unsigned f))
NONE(cudaGetSymbolAddress, (void** p, const void* s))
NONE(cudaGraphLaunch, (cudaGraphExec_t e, cudaStream_t s))
NONE(cudaGraphKernelNodeSetAttribute, (cudaGraphNode_t n, cudaLaunchAttributeID a, const cudaLaunchAttributeValue* v))
NONE(cudaGraphInstantiate, (cudaGraphExec_t* e, cudaGraph_t g, unsigned long long f))
NONE(cudaGraphExecDestroy, (cudaGraphExec_t e))
NONE(cudaGraphDestroy, (cudaGraph_t g))
NONE(cudaGraphCreate, (cudaGraph_t* g, unsigned f))
NONE(cudaGraphConditionalHandleCreate, (cudaGraphConditionalHandle* h, cudaGraph_t g, unsigned v, unsigned f))
NONE(cudaGraphAddNode, (cudaGraphNode_t* n, cudaGraph_t g, const cudaGraphNode_t* d, size_t k, struct cudaGraphNodeParams* p))
NONE(cudaGraphAddKernelNode, (cudaGraphNode_t* n, cudaGraph_t g, const cudaGraphNode_t* d, size_t k, const struct cudaKernelNodeParams* p))
