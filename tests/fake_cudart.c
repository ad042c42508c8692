/* A stand-in for the CUDA runtime's memory, stream and launch calls with two devices, preloaded in front of
 * it: device memory is host memory, launches do nothing. It keeps the current device, refuses a launch into
 * another device's stream as the runtime does, and logs every allocation (device, bytes) and pool call
 * (fake_log) and the launches' grids (fake_launches). The devices have fake_sms SMs. For tests of the
 * library's host code (test_device_calls.py). */
#include <cuda_runtime_api.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

int fake_sms = 148;
static int cur, last;
static char text[1 << 16], launches[1 << 16];
static void note(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  size_t n = strlen(text);
  vsnprintf(text + n, sizeof text - n, fmt, ap);
  va_end(ap);
}
const char* fake_log(void) { return text; }
const char* fake_launches(void) { return launches; }
void fake_clear(void) { text[0] = launches[0] = 0; }

struct CUstream_st { int device; };
struct CUevent_st { int device; };
struct CUmemPoolHandle_st { int device; };
static cudaError_t take(void** p, size_t n, const char* what) {
  *p = calloc(1, n + 4096);
  note("%s %d %zu\n", what, cur, n);
  return cudaSuccess;
}

cudaError_t cudaGetDevice(int* d) { *d = cur; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) {
  if (d < 0 || d > 1) return cudaErrorInvalidDevice;
  cur = d;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) { (void)a; (void)d; *v = fake_sms; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { int e = last; last = 0; return (cudaError_t)e; }
const char* cudaGetErrorString(cudaError_t e) { return e ? "refused" : "no error"; }
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) { (void)f; (void)a; (void)v; return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** args, size_t sm, cudaStream_t st) {
  (void)f; (void)b; (void)args; (void)sm;
  size_t n = strlen(launches);
  snprintf(launches + n, sizeof launches - n, "%u %u\n", g.x, g.y);
  if (st && st->device != cur) return (cudaError_t)(last = cudaErrorInvalidResourceHandle);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { (void)s; return take(p, 1 << 24, "symbol"); }
cudaError_t cudaMemcpyToSymbol(const void* s, const void* p, size_t n, size_t o, enum cudaMemcpyKind k) {
  (void)s; (void)p; (void)n; (void)o; (void)k;
  return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n, "malloc"); }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned f) { (void)f; *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned f) { (void)f; *d = h; return cudaSuccess; }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const struct cudaMemPoolProps* q) {
  *p = malloc(sizeof **p);
  (*p)->device = q->location.id;
  note("pool %d\n", q->location.id);
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, enum cudaMemPoolAttr a, void* v) { (void)p; (void)a; (void)v; return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t n) { note("trim %d to %zu\n", p->device, n); return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t st) {
  (void)st;
  *p = calloc(1, n);
  note("pooled %d\n", pool->device);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t st) { (void)st; free(p); return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) { (void)st; memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) { (void)k; memmove(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  (void)k; (void)st;
  memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, enum cudaMemcpyKind k, cudaStream_t st) {
  (void)k; (void)st;
  for (size_t y = 0; y < h; y++) memmove((char*)d + y * dp, (const char*)s + y * sp, w);
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) {
  (void)f;
  *s = malloc(sizeof **s);
  (*s)->device = cur;
  note("stream %d\n", cur);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s; (void)e; (void)f; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) {
  (void)f;
  *e = malloc(sizeof **e);
  (*e)->device = cur;
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
