/* A stand-in for the CUDA runtime, preloaded by test_host_launches.py: the
 * library's host code runs on the CPU, "device" memory is host memory,
 * launches are checked against the limits a device would enforce and
 * recorded, and no kernel runs.  Function attributes belong to the device
 * that is current when they are set, as on real devices. */
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

#define MAXK 4096
#define API __attribute__((visibility("default")))

static struct { const void* fn; const char* name; int smem[2], wide[2]; } kern[MAXK];
static int nkern, device, cluster_places = 1, attribute_fails;
static cudaError_t last;
static long allocs, launches, widest;
static unsigned long long bytes;

static cudaError_t fail(cudaError_t e) { return last = e; }
static int find(const void* fn) {
  for (int i = 0; i < nkern; ++i)
    if (kern[i].fn == fn) return i;
  return -1;
}

/* ---- the test's side ---- */
API void fake_set_device(int d) { device = d; }
API void fake_cluster_places(int n) { cluster_places = n; }
API void fake_attribute_fails(int on) { attribute_fails = on; }
API long fake_allocs(void) { return allocs; }
API unsigned long long fake_bytes(void) { return bytes; }
API long fake_launches(void) { return launches; }
API long fake_widest_cluster(void) { long w = widest; widest = 0; return w; }

/* ---- registration ---- */
API void** __cudaRegisterFatBinary(void* f) { return (void**)f; }
API void __cudaRegisterFatBinaryEnd(void** h) {}
API void __cudaUnregisterFatBinary(void** h) {}
API void __cudaRegisterVar(void** h, char* v, char* a, const char* n, int e, size_t s, int c, int g) {}
API void __cudaRegisterFunction(void** h, const char* fn, char* df, const char* name, int tl, uint3* a, uint3* b,
                                dim3* c, dim3* d, int* w) {
  kern[nkern].fn = fn;
  kern[nkern++].name = name;
}

/* ---- launches ---- */
static dim3 cfg_grid, cfg_block;
static size_t cfg_smem;
static cudaStream_t cfg_stream;
API unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, struct CUstream_st* st) {
  cfg_grid = g; cfg_block = b; cfg_smem = s; cfg_stream = st;
  return 0;
}
API cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) {
  *g = cfg_grid; *b = cfg_block; *s = cfg_smem; *(cudaStream_t*)st = cfg_stream;
  return cudaSuccess;
}
static cudaError_t launch(const void* fn, size_t smem, unsigned cluster) {
  const int k = find(fn);
  if (k < 0) return fail(cudaErrorInvalidDeviceFunction);
  if (smem > 48 * 1024 && smem > (size_t)kern[k].smem[device]) return fail(cudaErrorInvalidValue);
  if (cluster > 8 && (!kern[k].wide[device] || cluster_places == 0)) return fail(cudaErrorInvalidClusterSize);
  if (cluster > widest) widest = cluster;
  ++launches;
  return cudaSuccess;
}
API cudaError_t cudaLaunchKernel(const void* fn, dim3 g, dim3 b, void** a, size_t s, cudaStream_t st) {
  return launch(fn, s, 1);
}
API cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void** a) {
  unsigned cluster = 1;
  for (unsigned i = 0; i < c->numAttrs; ++i)
    if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cluster = c->attrs[i].val.clusterDim.x;
  return launch(fn, c->dynamicSmemBytes, cluster);
}
API cudaError_t cudaFuncSetAttribute(const void* fn, enum cudaFuncAttribute at, int v) {
  const int k = find(fn);
  if (k < 0) return fail(cudaErrorInvalidDeviceFunction);
  if (at == cudaFuncAttributeMaxDynamicSharedMemorySize) kern[k].smem[device] = v;
  if (at == cudaFuncAttributeNonPortableClusterSizeAllowed) {
    if (attribute_fails) return fail(cudaErrorInvalidValue);
    kern[k].wide[device] = v;
  }
  return cudaSuccess;
}
API cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void* fn) {
  memset(a, 0, sizeof *a);
  return cudaSuccess;
}
API cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* fn, int b, size_t s,
                                                                       unsigned f) {
  *n = 4;
  return cudaSuccess;
}
API cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* fn, const cudaLaunchConfig_t* c) {
  const int k = find(fn);
  if (k < 0 || !kern[k].wide[device]) return fail(cudaErrorInvalidClusterSize);
  *n = cluster_places;
  return cudaSuccess;
}

/* ---- memory, streams, the device ---- */
API cudaError_t cudaMalloc(void** p, size_t n) {
  *p = malloc(n);
  if (!*p) return fail(cudaErrorMemoryAllocation);
  ++allocs;
  bytes += n;
  return cudaSuccess;
}
API cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
API cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) { memcpy(d, s, n); return cudaSuccess; }
API cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  memcpy(d, s, n);
  return cudaSuccess;
}
API cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
API cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) { memset(d, v, n); return cudaSuccess; }
API cudaError_t cudaGetSymbolAddress(void** p, const void* s) { return fail(cudaErrorInvalidSymbol); }
API cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
API cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 227 * 1024 : 0;
  return cudaSuccess;
}
API cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
API cudaError_t cudaGetLastError(void) { cudaError_t e = last; last = cudaSuccess; return e; }
API const char* cudaGetErrorString(cudaError_t e) { return "fake"; }
API cudaError_t cudaGetDriverEntryPoint(const char* n, void** p, unsigned long long f,
                                        enum cudaDriverEntryPointQueryResult* q) {
  return fail(cudaErrorNotSupported);
}
static char handle;
API cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) { *s = (cudaStream_t)&handle; return cudaSuccess; }
API cudaError_t cudaStreamDestroy(cudaStream_t s) { return cudaSuccess; }
API cudaError_t cudaStreamSynchronize(cudaStream_t s) { return cudaSuccess; }
API cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { return cudaSuccess; }
API cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) { *e = (cudaEvent_t)&handle; return cudaSuccess; }
API cudaError_t cudaEventDestroy(cudaEvent_t e) { return cudaSuccess; }
API cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return cudaSuccess; }
