/* A stand-in for the CUDA runtime and cuFFT entry points that the library
 * calls, preloaded on a machine without a GPU.  Nothing runs on a device: every
 * launch, copy, event and wait is written to the file named by STREAM_LOG, one
 * line each, so that a test can ask which operation is ordered after which.
 * "Device" memory is host memory filled with 0x3f (positive as a float or a
 * double); copies are carried out, and sets of up to 64 KB (a mesh stays positive). */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

typedef struct { unsigned x, y, z; } dim3;
typedef void* ptr;

static void put(const char* fmt, const void* a, const void* b, const char* s) {
  static FILE* f;
  if (!f && !(f = fopen(getenv("STREAM_LOG"), "w"))) abort();
  fprintf(f, fmt, (unsigned long)a, (unsigned long)b, s);
  fflush(f);
}
static ptr fresh(void) { return malloc(64); } /* a handle */

/* kernels: name and launch */
static struct { const void* fun; char name[256]; } kern[1024];
static int nkern;
static struct { dim3 g, b; size_t s; ptr st; } cfg;
void** __cudaRegisterFatBinary(void* p) { return (void**)fresh(); }
void __cudaRegisterFatBinaryEnd(void** h) {}
void __cudaUnregisterFatBinary(void** h) {}
void __cudaRegisterVar(void** h, char* v, char* d, const char* n, int e, size_t s, int c, int g) {}
void __cudaRegisterFunction(void** h, const char* fun, char* d, const char* name, int l, void* t, void* b, void* bd,
                            void* gd, int* w) {
  kern[nkern].fun = fun;
  strncpy(kern[nkern++].name, name, 255);
}
int __cudaGetKernel(ptr* k, const void* fun) {
  *k = (ptr)fun;
  return 0;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, ptr st) {
  cfg.g = g, cfg.b = b, cfg.s = s, cfg.st = st;
  return 0;
}
int __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, ptr* st) {
  *g = cfg.g, *b = cfg.b, *s = cfg.s, *st = cfg.st;
  return 0;
}
int __cudaLaunchKernel(ptr k, dim3 g, dim3 b, void** args, size_t s, ptr st) {
  for (int i = 0; i < nkern; i++)
    if (kern[i].fun == k) put("op %lu %lu %s\n", st, 0, kern[i].name);
  return 0;
}

/* memory */
int cudaMalloc(ptr* p, size_t n) { return (*p = malloc(n + 64)) ? (memset(*p, 0x3f, n + 64), 0) : 2; }
int cudaMallocHost(ptr* p, size_t n) { return (*p = calloc(1, n)) ? 0 : 2; }
int cudaFree(ptr p) { return free(p), 0; }
int cudaFreeHost(ptr p) { return free(p), 0; }
int cudaMemcpy(ptr d, const void* s, size_t n, int k) { return memmove(d, s, n), 0; }
int cudaMemset(ptr d, int v, size_t n) { return memset(d, v, n), 0; }
int cudaMemcpyAsync(ptr d, const void* s, size_t n, int k, ptr st) {
  put("op %lu %lu %s\n", st, d, "memcpy");
  return memmove(d, s, n), 0;
}
int cudaMemsetAsync(ptr d, int v, size_t n, ptr st) {
  put("op %lu %lu %s\n", st, d, "memset");
  return n <= 1 << 16 ? memset(d, v, n) : d, 0;
}
int cudaMemcpy2DAsync(ptr d, size_t dp, const void* s, size_t sp, size_t w, size_t h, int k, ptr st) {
  put("op %lu %lu %s\n", st, d, "memcpy2D");
  for (size_t i = 0; i < h; i++) memmove((char*)d + i * dp, (const char*)s + i * sp, w);
  return 0;
}
int cudaGetSymbolAddress(ptr* p, const void* s) { return (*p = calloc(1, 1 << 22)) ? 0 : 2; }

/* streams, events, graphs */
int cudaStreamCreateWithFlags(ptr* s, unsigned f) { return *s = fresh(), 0; }
int cudaStreamCreateWithPriority(ptr* s, unsigned f, int p) { return *s = fresh(), 0; }
int cudaDeviceGetStreamPriorityRange(int* a, int* b) { return *a = *b = 0, 0; }
int cudaStreamDestroy(ptr s) { return 0; }
int cudaEventCreate(ptr* e) { return *e = fresh(), 0; }
int cudaEventCreateWithFlags(ptr* e, unsigned f) { return *e = fresh(), 0; }
int cudaEventDestroy(ptr e) { return 0; }
int cudaEventElapsedTime(float* ms, ptr a, ptr b) { return *ms = 1.f, 0; }
int cudaEventRecord(ptr e, ptr s) { return put("record %lu %lu %s\n", s, e, "-"), 0; }
int cudaStreamWaitEvent(ptr s, ptr e, unsigned f) { return put("wait %lu %lu %s\n", s, e, "-"), 0; }
int cudaEventSynchronize(ptr e) { return put("hostwait %lu %lu %s\n", 0, e, "-"), 0; }
int cudaStreamSynchronize(ptr s) { return put("sync %lu %lu %s\n", s, 0, "-"), 0; }
int cudaDeviceSynchronize(void) { return put("syncall %lu %lu %s\n", 0, 0, "-"), 0; }
int cudaStreamBeginCapture(ptr s, int m) { return 0; }
int cudaStreamEndCapture(ptr s, ptr* g) { return *g = fresh(), 0; }
int cudaGraphInstantiate(ptr* x, ptr g, unsigned long long f) { return *x = fresh(), 0; }
int cudaGraphLaunch(ptr x, ptr s) { return 0; }
int cudaGraphDestroy(ptr g) { return 0; }
int cudaGraphExecDestroy(ptr x) { return 0; }

/* the device */
int cudaSetDevice(int d) { return 0; }
int cudaGetDevice(int* d) { return *d = 0, 0; }
int cudaGetDeviceCount(int* n) { return *n = 1, 0; }
int cudaDeviceGetAttribute(int* v, int a, int d) { /* multiprocessors */
  const char* n = getenv("STREAM_SMS");
  return *v = n ? atoi(n) : 152, 0;
}
int cudaFuncGetAttributes(void* a, const void* f) { /* sizes, then threads, registers, PTX and binary version */
  const int v[4] = {1024, 32, 103, 103};
  return memset(a, 0, 128), memcpy((char*)a + 3 * sizeof(size_t), v, sizeof v), 0;
}
int cudaFuncSetAttribute(const void* f, int a, int v) { return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int b, size_t s, unsigned fl) {
  return *n = 1, 0;
}
int cudaGetLastError(void) { return 0; }
int cudaPeekAtLastError(void) { return 0; }
const char* cudaGetErrorString(int e) { return "error"; }

/* cuFFT */
static ptr plan_stream[64];
static int nplan;
int cufftCreate(int* h) { return *h = ++nplan % 64, 0; }
int cufftDestroy(int h) { return 0; }
int cufftSetAutoAllocation(int h, int a) { return 0; }
int cufftMakePlan3d(int h, int x, int y, int z, int t, size_t* w) { return *w = 1 << 16, 0; }
int cufftMakePlanMany(int h, int r, int* n, int* i, int is, int id, int* o, int os, int od, int t, int b, size_t* w) {
  return *w = 1 << 16, 0;
}
int cufftPlan3d(int* h, int x, int y, int z, int t) { return cufftCreate(h); }
int cufftSetWorkArea(int h, ptr w) { return 0; }
int cufftSetStream(int h, ptr s) { return plan_stream[h] = s, 0; }
int cufftExecC2R(int h, ptr i, ptr o) { return put("op %lu %lu %s\n", plan_stream[h], o, "c2r"), 0; }
int cufftExecR2C(int h, ptr i, ptr o) { return put("op %lu %lu %s\n", plan_stream[h], o, "r2c"), 0; }
