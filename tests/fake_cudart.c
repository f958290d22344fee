/* A CUDA runtime without a GPU, for the host side's use of devices: memory is
 * the host's, kernels are not run, and a stream or event remembers the device
 * that was current when it was created. As in the real runtime, a kernel
 * launch or an event record on a stream of another device than the calling
 * thread's current one is refused (cudaErrorInvalidResourceHandle), while
 * copies may go to any stream. fake_malloc_device tells where an allocation
 * was made, fake_launches how many kernels were launched. */
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#define DEVICES 2
#define MAX_ALLOCS 65536
enum { SUCCESS = 0, INVALID_VALUE = 1, INVALID_DEVICE = 101, BAD_HANDLE = 400,
       NOT_SUPPORTED = 801 };

typedef struct { int device; } Handle; /* a stream or an event */
typedef struct { unsigned x, y, z; } Dim3;
typedef struct {
  Dim3 grid, block;
  size_t smem;
  Handle* stream;
  void* attrs;
  unsigned num_attrs;
} LaunchConfig;

static __thread int current;
static int launches, last_error;
static struct { char* p; size_t n; int device; } allocs[MAX_ALLOCS];
static int num_allocs;
static LaunchConfig pushed;

static int Fail(int e) {
  last_error = e;
  return e;
}
int fake_launches(void) { return launches; }
int fake_malloc_device(const void* p) {
  for (int i = 0; i < num_allocs; ++i) {
    if (allocs[i].p && (const char*)p >= allocs[i].p &&
        (const char*)p < allocs[i].p + allocs[i].n) {
      return allocs[i].device;
    }
  }
  return -1;
}

int cudaGetDeviceCount(int* n) { *n = DEVICES; return SUCCESS; }
int cudaGetDevice(int* d) { *d = current; return SUCCESS; }
int cudaSetDevice(int d) {
  if (d < 0 || d >= DEVICES) return Fail(INVALID_DEVICE);
  current = d;
  return SUCCESS;
}
int cudaDeviceGetAttribute(int* v, int attr, int d) {
  (void)attr, (void)d;
  *v = 148;
  return SUCCESS;
}
const char* cudaGetErrorString(int e) {
  return e == BAD_HANDLE ? "invalid resource handle" : "error";
}
int cudaGetLastError(void) {
  const int e = last_error;
  last_error = SUCCESS;
  return e;
}

int cudaMalloc(void** p, size_t n) {
  *p = calloc(1, n);
  if (*p && num_allocs < MAX_ALLOCS) {
    allocs[num_allocs].p = *p;
    allocs[num_allocs].n = n;
    allocs[num_allocs++].device = current;
  }
  return *p ? SUCCESS : Fail(2);
}
int cudaFree(void* p) {
  for (int i = 0; p && i < num_allocs; ++i) {
    if (allocs[i].p == p) allocs[i].p = NULL;
  }
  free(p);
  return SUCCESS;
}
int cudaHostAlloc(void** p, size_t n, unsigned flags) {
  (void)flags;
  *p = calloc(1, n);
  return SUCCESS;
}
int cudaFreeHost(void* p) { free(p); return SUCCESS; }
int cudaMemcpy(void* d, const void* s, size_t n, int kind) {
  (void)kind;
  memmove(d, s, n);
  return SUCCESS;
}
int cudaMemcpyAsync(void* d, const void* s, size_t n, int kind, Handle* st) {
  (void)st;
  return cudaMemcpy(d, s, n, kind);
}
int cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w,
                 size_t h, int kind) {
  (void)kind;
  for (size_t y = 0; y < h; ++y) {
    memmove((char*)d + y * dp, (const char*)s + y * sp, w);
  }
  return SUCCESS;
}
int cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w,
                      size_t h, int kind, Handle* st) {
  (void)st;
  return cudaMemcpy2D(d, dp, s, sp, w, h, kind);
}
int cudaMemsetAsync(void* p, int v, size_t n, Handle* st) {
  (void)st;
  memset(p, v, n);
  return SUCCESS;
}
int cudaMemcpyToSymbol(const void* sym, const void* s, size_t n, size_t off,
                       int kind) {
  (void)sym, (void)s, (void)n, (void)off, (void)kind;
  return SUCCESS;
}
int cudaGetSymbolAddress(void** p, const void* sym) {
  (void)sym, (void)p;
  return Fail(NOT_SUPPORTED);
}
int cudaPointerGetAttributes(void* a, const void* p) {
  (void)a, (void)p;
  return Fail(INVALID_VALUE);
}

static int NewHandle(Handle** h) {
  *h = malloc(sizeof(Handle));
  (*h)->device = current;
  return SUCCESS;
}
int cudaStreamCreateWithFlags(Handle** s, unsigned f) {
  (void)f;
  return NewHandle(s);
}
int cudaStreamDestroy(Handle* s) { free(s); return SUCCESS; }
int cudaStreamSynchronize(Handle* s) { (void)s; return SUCCESS; }
int cudaStreamWaitEvent(Handle* s, Handle* e, unsigned f) {
  (void)s, (void)e, (void)f;
  return SUCCESS;
}
int cudaEventCreate(Handle** e) { return NewHandle(e); }
int cudaEventCreateWithFlags(Handle** e, unsigned f) {
  (void)f;
  return NewHandle(e);
}
int cudaEventDestroy(Handle* e) { free(e); return SUCCESS; }
int cudaEventSynchronize(Handle* e) { (void)e; return SUCCESS; }
int cudaEventElapsedTime(float* ms, Handle* a, Handle* b) {
  (void)a, (void)b;
  *ms = 0.0f;
  return SUCCESS;
}
int cudaEventRecord(Handle* e, Handle* s) {
  return s && s->device != e->device ? Fail(BAD_HANDLE) : SUCCESS;
}

static int Launch(const Handle* s) {
  if (s && s->device != current) return Fail(BAD_HANDLE);
  ++launches;
  return SUCCESS;
}
int cudaLaunchKernel(const void* f, Dim3 g, Dim3 b, void** args, size_t smem,
                     Handle* s) {
  (void)f, (void)g, (void)b, (void)args, (void)smem;
  return Launch(s);
}
int cudaLaunchKernelExC(const LaunchConfig* c, const void* f, void** args) {
  (void)f, (void)args;
  return Launch(c->stream);
}
int cudaFuncSetAttribute(const void* f, int attr, int v) {
  (void)f, (void)attr, (void)v;
  return SUCCESS;
}
int cudaGetDriverEntryPoint(const char* name, void** p, unsigned long long f,
                            int* status) {
  (void)name, (void)f;
  *p = NULL;
  if (status) *status = 1; /* not found */
  return SUCCESS;
}
int cudaStreamBeginCapture(Handle* s, int mode) {
  (void)s, (void)mode;
  return Fail(NOT_SUPPORTED);
}
int cudaStreamEndCapture(Handle* s, void** g) {
  (void)s, (void)g;
  return Fail(NOT_SUPPORTED);
}
int cudaGraphInstantiate(void** e, void* g, unsigned long long f) {
  (void)e, (void)g, (void)f;
  return Fail(NOT_SUPPORTED);
}
int cudaGraphLaunch(void* e, Handle* s) {
  (void)e, (void)s;
  return Fail(NOT_SUPPORTED);
}
int cudaGraphDestroy(void* g) { (void)g; return SUCCESS; }
int cudaGraphExecDestroy(void* e) { (void)e; return SUCCESS; }

/* What the compiler's host code calls. */
void** __cudaRegisterFatBinary(void* b) {
  static void* handle;
  (void)b;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
char __cudaInitModule(void** h) { (void)h; return 1; }
void __cudaRegisterFunction(void** h, const char* f, char* df,
                            const char* name, int tl, void* tid, void* bid,
                            Dim3* bd, Dim3* gd, int* ws) {
  (void)h, (void)f, (void)df, (void)name, (void)tl, (void)tid, (void)bid;
  (void)bd, (void)gd, (void)ws;
}
void __cudaRegisterVar(void** h, char* v, char* da, const char* name, int ext,
                       size_t n, int c, int g) {
  (void)h, (void)v, (void)da, (void)name, (void)ext, (void)n, (void)c, (void)g;
}
unsigned __cudaPushCallConfiguration(Dim3 g, Dim3 b, size_t smem, Handle* s) {
  pushed.grid = g, pushed.block = b, pushed.smem = smem, pushed.stream = s;
  return 0;
}
int __cudaPopCallConfiguration(Dim3* g, Dim3* b, size_t* smem, void* s) {
  *g = pushed.grid, *b = pushed.block, *smem = pushed.smem;
  *(Handle**)s = pushed.stream;
  return SUCCESS;
}
