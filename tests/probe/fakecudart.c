/* A CUDA runtime without a device, for the library's host logic: preloaded in front of libcudart, it
 * keeps memory on the host, runs no kernel but the one that copies words to the host, counts launches
 * and captures, and refuses the launches it is told to.  (TEST INFRASTRUCTURE ONLY) */
#include <stdlib.h>
#include <string.h>

typedef int err_t;
typedef void *stream_t;
typedef struct { unsigned x, y, z; } dim_t;
typedef struct { dim_t grid, block; size_t smem; stream_t stream; void *attrs; unsigned n; } config_t;

enum { MOST = 4096 };
static const void *fun[MOST];
static const char *name[MOST];
static int n_funs, last, captures, graphs, launches, refused;
static char refuse[128];

/* the test's side */
void fake_refuse(const char *kernel) { strncpy(refuse, kernel, sizeof refuse - 1); }
int fake_captures(void) { return captures; }
int fake_graph_launches(void) { return graphs; }
int fake_launches(void) { return launches; }
int fake_refused(void) { return refused; }

static err_t launch(const void *f, void **args) {
  const char *s = "";
  for (int k = 0; k < n_funs; ++k)
    if (fun[k] == f) s = name[k];
  if (refuse[0] && strstr(s, refuse)) {
    ++refused;
    return last = 1; /* cudaErrorInvalidValue */
  }
  ++launches;
  if (strstr(s, "k_words_out")) memcpy(*(void **)args[1], *(void **)args[0], 4 * (size_t)*(int *)args[2]);
  return 0;
}
void **__cudaRegisterFatBinary(void *p) { return (void **)p; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterVar(void **h, char *v, char *a, const char *s, int e, size_t z, int c, int g) {
  (void)h, (void)v, (void)a, (void)s, (void)e, (void)z, (void)c, (void)g;
}
void __cudaRegisterFunction(void **h, const char *f, char *d, const char *s, int l, void *t, void *b, void *bd, void *gd,
                            int *w) {
  (void)h, (void)d, (void)l, (void)t, (void)b, (void)bd, (void)gd, (void)w;
  if (n_funs < MOST) fun[n_funs] = f, name[n_funs++] = s;
}
static config_t pushed;
unsigned __cudaPushCallConfiguration(dim_t g, dim_t b, size_t m, void *s) {
  pushed.grid = g, pushed.block = b, pushed.smem = m, pushed.stream = s;
  return 0;
}
err_t __cudaPopCallConfiguration(dim_t *g, dim_t *b, size_t *m, void *s) {
  *g = pushed.grid, *b = pushed.block, *m = pushed.smem, *(void **)s = pushed.stream;
  return 0;
}
err_t __cudaGetKernel(const void **k, const void *f) { return *k = f, 0; }
err_t __cudaLaunchKernel(const void *k, dim_t g, dim_t b, void **a, size_t m, stream_t s) {
  (void)g, (void)b, (void)m, (void)s;
  return launch(k, a);
}
err_t cudaLaunchKernelExC(const config_t *c, const void *f, void **a) { return (void)c, launch(f, a); }
err_t cudaGetLastError(void) { const err_t e = last; return last = 0, e; }
const char *cudaGetErrorString(err_t e) { return e ? "refused by the test" : "no error"; }

err_t cudaMalloc(void **p, size_t n) { return (*p = calloc(1, n ? n : 1)) ? 0 : 2; }
err_t cudaHostAlloc(void **p, size_t n, unsigned f) { return (void)f, cudaMalloc(p, n); }
err_t cudaFree(void *p) { return free(p), 0; }
err_t cudaFreeHost(void *p) { return free(p), 0; }
err_t cudaMemcpy(void *d, const void *s, size_t n, int k) { return (void)k, memmove(d, s, n), 0; }
err_t cudaMemcpyAsync(void *d, const void *s, size_t n, int k, stream_t t) { return (void)t, cudaMemcpy(d, s, n, k); }
err_t cudaMemset(void *d, int v, size_t n) { return memset(d, v, n), 0; }
err_t cudaMemsetAsync(void *d, int v, size_t n, stream_t t) { return (void)t, cudaMemset(d, v, n); }
err_t cudaMemcpyToSymbol(const void *d, const void *s, size_t n, size_t o, int k) {
  return (void)d, (void)s, (void)n, (void)o, (void)k, 0;
}
err_t cudaGetSymbolAddress(void **p, const void *s) { return (void)p, (void)s, last = 13; }
err_t cudaPointerGetAttributes(void *a, const void *p) { return (void)a, (void)p, last = 1; }

err_t cudaGetDeviceCount(int *n) { return *n = 1, 0; }
err_t cudaGetDevice(int *d) { return *d = 0, 0; }
err_t cudaSetDevice(int d) { return (void)d, 0; }
err_t cudaDeviceGetAttribute(int *v, int a, int d) { return (void)a, (void)d, *v = 152, 0; }
err_t cudaDeviceGetStreamPriorityRange(int *l, int *m) { return *l = 0, *m = -1, 0; }
err_t cudaDeviceSynchronize(void) { return 0; }
err_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int b, size_t m, unsigned g) {
  return (void)f, (void)b, (void)m, (void)g, *n = 2, 0;
}
err_t cudaFuncSetAttribute(const void *f, int a, int v) { return (void)f, (void)a, (void)v, 0; }
err_t cudaGetDriverEntryPointByVersion(const char *s, void **p, unsigned v, unsigned long long f, int *q) {
  return (void)s, (void)p, (void)v, (void)f, (void)q, last = 1;
}

static err_t handle(void **h) { return (*h = malloc(1)) ? 0 : 2; }
err_t cudaStreamCreateWithFlags(stream_t *s, unsigned f) { return (void)f, handle(s); }
err_t cudaStreamCreateWithPriority(stream_t *s, unsigned f, int p) { return (void)f, (void)p, handle(s); }
err_t cudaStreamDestroy(stream_t s) { return free(s), 0; }
err_t cudaStreamSynchronize(stream_t s) { return (void)s, 0; }
err_t cudaStreamWaitEvent(stream_t s, void *e, unsigned f) { return (void)s, (void)e, (void)f, 0; }
err_t cudaEventCreate(void **e) { return handle(e); }
err_t cudaEventCreateWithFlags(void **e, unsigned f) { return (void)f, handle(e); }
err_t cudaEventDestroy(void *e) { return free(e), 0; }
err_t cudaEventRecord(void *e, stream_t s) { return (void)e, (void)s, 0; }
err_t cudaEventSynchronize(void *e) { return (void)e, 0; }
err_t cudaEventElapsedTime(float *t, void *a, void *b) { return (void)a, (void)b, *t = 0.0f, 0; }
err_t cudaStreamBeginCapture(stream_t s, int m) { return (void)s, (void)m, ++captures, 0; }
err_t cudaStreamEndCapture(stream_t s, void **g) { return (void)s, handle(g); }
err_t cudaGraphInstantiate(void **x, void *g, unsigned long long f) { return (void)g, (void)f, handle(x); }
err_t cudaGraphDestroy(void *g) { return free(g), 0; }
err_t cudaGraphExecDestroy(void *x) { return free(x), 0; }
err_t cudaGraphLaunch(void *x, stream_t s) { return (void)x, (void)s, ++graphs, 0; }
