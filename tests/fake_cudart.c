/* A stand-in for the CUDA runtime that runs nothing: it gives out host addresses as device memory and
 * writes every allocation, launch, event record and event wait of liblh.so to the file that
 * FAKE_CUDART_LOG names. Preloaded into a process without a GPU, it shows what the host code asks of
 * the device: which buffers a launch gets, on which stream, after which events. A line each:
 *   A address bytes | F address | L kernel stream gx gy gz bx by bz smem [arguments] |
 *   R event stream | W stream event
 * FAKE_CUDART_ARGS ("kernel:n,kernel:n") names the kernels whose first n arguments are logged; these
 * must be pointers. */
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

typedef struct { unsigned x, y, z; } dim3_t;

static FILE *out(void) {
  static FILE *f;
  if (!f) {
    const char *p = getenv("FAKE_CUDART_LOG");
    f = p ? fopen(p, "w") : stderr;
    if (!f) abort();
    setvbuf(f, NULL, _IOLBF, 0);
  }
  return f;
}

/* ---- kernels ---- */
static struct { const void *fun; const char *name; } kernels[8192];
static int nkernels;
static dim3_t cfg_grid, cfg_block;
static size_t cfg_smem;
static void *cfg_stream;

void **__cudaRegisterFatBinary(void *fat) { (void)fat; static void *handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterVar(void **h, char *var, char *addr, const char *name, int ext, size_t size, int constant, int global) {
  (void)h; (void)var; (void)addr; (void)name; (void)ext; (void)size; (void)constant; (void)global;
}
void __cudaRegisterFunction(void **h, const char *fun, char *dev, const char *name, int limit, void *tid, void *bid,
                            void *bdim, void *gdim, int *wsize) {
  (void)h; (void)dev; (void)limit; (void)tid; (void)bid; (void)bdim; (void)gdim; (void)wsize;
  if (nkernels == 8192) abort();
  kernels[nkernels].fun = fun;
  kernels[nkernels++].name = name;
}
int __cudaGetKernel(void **kernel, const void *fun) { *kernel = (void *)fun; return 0; }
unsigned __cudaPushCallConfiguration(dim3_t grid, dim3_t block, size_t smem, void *stream) {
  cfg_grid = grid; cfg_block = block; cfg_smem = smem; cfg_stream = stream;
  return 0;
}
int __cudaPopCallConfiguration(dim3_t *grid, dim3_t *block, size_t *smem, void *stream) {
  *grid = cfg_grid; *block = cfg_block; *smem = cfg_smem; *(void **)stream = cfg_stream;
  return 0;
}
int __cudaLaunchKernel(void *kernel, dim3_t g, dim3_t b, void **args, size_t smem, void *stream) {
  const char *name = "?";
  for (int i = 0; i < nkernels; ++i)
    if (kernels[i].fun == kernel) name = kernels[i].name;
  fprintf(out(), "L %s %p %u %u %u %u %u %u %zu", name, stream, g.x, g.y, g.z, b.x, b.y, b.z, smem);
  const char *want = getenv("FAKE_CUDART_ARGS");
  while (want && *want) {
    char key[64];
    int n = 0, len = 0;
    if (sscanf(want, "%63[^:]:%d%n", key, &n, &len) != 2) break;
    if (strstr(name, key))
      for (int i = 0; i < n; ++i) fprintf(out(), " %p", *(void **)args[i]);
    want += len;
    if (*want == ',') ++want;
  }
  fprintf(out(), "\n");
  return 0;
}

/* ---- memory: addresses only, nothing is copied ---- */
int cudaMalloc(void **p, size_t n) {
  *p = malloc(n);
  fprintf(out(), "A %p %zu\n", *p, n);
  return *p ? 0 : 2;
}
int cudaFree(void *p) { fprintf(out(), "F %p\n", p); free(p); return 0; }
int cudaMemcpy(void *d, const void *s, size_t n, int k) { (void)s; if (k == 2) memset(d, 0, n); return 0; }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int k, void *st) { (void)st; return cudaMemcpy(d, s, n, k); }
int cudaMemset(void *p, int v, size_t n) { (void)p; (void)v; (void)n; return 0; }
int cudaMemsetAsync(void *p, int v, size_t n, void *st) { (void)st; return cudaMemset(p, v, n); }
int cudaGetSymbolAddress(void **p, const void *s) { *p = (void *)s; return 0; }

/* ---- streams, events, graphs ---- */
static int fresh(void **p) { static uintptr_t n; *p = (void *)(0x1000 + 16 * ++n); return 0; }
int cudaStreamCreateWithFlags(void **s, unsigned f) { (void)f; return fresh(s); }
int cudaStreamDestroy(void *s) { (void)s; return 0; }
int cudaStreamSynchronize(void *s) { (void)s; return 0; }
int cudaStreamBeginCapture(void *s, int m) { (void)s; (void)m; return 0; }
int cudaStreamEndCapture(void *s, void **g) { (void)s; return fresh(g); }
int cudaEventCreate(void **e) { return fresh(e); }
int cudaEventCreateWithFlags(void **e, unsigned f) { (void)f; return fresh(e); }
int cudaEventDestroy(void *e) { (void)e; return 0; }
int cudaEventElapsedTime(float *ms, void *a, void *b) { (void)a; (void)b; *ms = 1.0f; return 0; }
int cudaEventRecord(void *e, void *s) { fprintf(out(), "R %p %p\n", e, s); return 0; }
int cudaStreamWaitEvent(void *s, void *e, unsigned f) { (void)f; fprintf(out(), "W %p %p\n", s, e); return 0; }
int cudaGraphInstantiate(void **x, void *g, unsigned long long f) { (void)g; (void)f; return fresh(x); }
int cudaGraphLaunch(void *x, void *s) { (void)x; (void)s; return 0; }
int cudaGraphGetNodes(void *g, void **nodes, size_t *n) { (void)g; (void)nodes; *n = 1; return 0; }
int cudaGraphDestroy(void *g) { (void)g; return 0; }
int cudaGraphExecDestroy(void *x) { (void)x; return 0; }

/* ---- device and errors ---- */
int cudaGetDevice(int *d) { *d = 0; return 0; }
int cudaDeviceGetAttribute(int *v, int a, int d) { (void)a; (void)d; *v = 232448; return 0; } /* shared memory of a block */
int cudaFuncSetAttribute(const void *f, int a, int v) { (void)f; (void)a; (void)v; return 0; }
int cudaFuncGetAttributes(void *a, const void *f) { (void)a; (void)f; return 1; }
int cudaGetLastError(void) { return 0; }
const char *cudaGetErrorString(int e) { (void)e; return "stand-in runtime"; }
