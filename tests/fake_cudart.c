/*
 * A stand-in for the CUDA runtime, preloaded into a child process — TEST
 * INFRASTRUCTURE ONLY.  The library's host code runs as it is, on a machine without a
 * GPU: "device" memory is host memory, kernels do nothing but are counted by name, and
 * calls fail where a test asks for it.  The one kernel with an effect is the step's
 * finalize: it writes its log row (a NaN wall stress where the lost word is set) and
 * advances the row, as the device code does.
 */
#include <math.h>
#include <stddef.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

enum { OK = 0, ENOMEM_ = 2, KERNELS = 512, BLOCKS = 4096 };
typedef struct { unsigned x, y, z; } dim3_;

static struct { const void *fn; char name[256]; long launches; } kernels[KERNELS];
static int nkernels;
static struct { void *p; size_t n; } blocks[BLOCKS];
static size_t limit = (size_t)64 << 30, used;
static int last_error, capturing;
static long graph_launches, instantiated, fail_graph_launch;
static unsigned lost;
static double stress;
static dim3_ cfg_grid, cfg_block;
static size_t cfg_smem;
static void *cfg_stream;

/* what the tests set and read */
void fake_limit(size_t bytes) { limit = bytes; }
size_t fake_used(void) { return used; }
void fake_lost(unsigned on) { lost = on; }
void fake_stress(double v) { stress = v; }
void fake_fail_graph_launch(long on) { fail_graph_launch = on; }
long fake_graph_launches(void) { return graph_launches; }
long fake_instantiated(void) { return instantiated; }
long fake_launches(const char *part) {
  long n = 0;
  for (int k = 0; k < nkernels; k++)
    if (strstr(kernels[k].name, part)) n += kernels[k].launches;
  return n;
}

static int err(int e) {
  if (e) last_error = e;
  return e;
}

/* ---- registration and launches */
void **__cudaRegisterFatBinary(void *f) { (void)f; static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterVar(void **h, char *v, char *a, const char *n, int e, size_t s, int c, int g) {
  (void)h; (void)v; (void)a; (void)n; (void)e; (void)s; (void)c; (void)g;
}
void __cudaRegisterFunction(void **h, const char *fn, char *dev, const char *name, int lim, void *t, void *b, void *bd,
                            void *gd, int *w) {
  (void)h; (void)dev; (void)lim; (void)t; (void)b; (void)bd; (void)gd; (void)w;
  if (nkernels < KERNELS) {
    kernels[nkernels].fn = fn;
    strncpy(kernels[nkernels++].name, name, 255);
  }
}
unsigned __cudaPushCallConfiguration(dim3_ g, dim3_ b, size_t smem, void *stream) {
  cfg_grid = g; cfg_block = b; cfg_smem = smem; cfg_stream = stream;
  return 0;
}
int __cudaPopCallConfiguration(dim3_ *g, dim3_ *b, size_t *smem, void **stream) {
  *g = cfg_grid; *b = cfg_block; *smem = cfg_smem; *stream = cfg_stream;
  return 0;
}
int cudaLaunchKernel(const void *fn, dim3_ g, dim3_ b, void **args, size_t smem, void *stream) {
  (void)g; (void)b; (void)smem; (void)stream;
  for (int k = 0; k < nkernels; k++) {
    if (kernels[k].fn != fn) continue;
    kernels[k].launches++;
    if (!capturing && strstr(kernels[k].name, "finalize2_kernel")) {
      double *row = *(double **)args[1]; /* rows of 8 doubles, the stress the seventh */
      unsigned *counter = *(unsigned **)args[7];
      if (lost) counter[2] = 1;
      row += (size_t)counter[1]++ * 8;
      memset(row, 0, 64);
      row[6] = counter[2] ? NAN : stress;
    }
    return OK;
  }
  return err(98); /* not a registered kernel */
}
int cudaFuncSetAttribute(const void *f, int a, int v) { (void)f; (void)a; (void)v; return OK; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int b, size_t s, unsigned fl) {
  (void)f; (void)b; (void)s; (void)fl;
  *n = 1;
  return OK;
}

/* ---- memory */
static int get(void **p, size_t n) {
  if (used + n > limit) return err(ENOMEM_);
  for (int k = 0; k < BLOCKS; k++)
    if (!blocks[k].p) {
      if (!(*p = calloc(n ? n : 1, 1))) return err(ENOMEM_);
      blocks[k].p = *p;
      blocks[k].n = n;
      used += n;
      return OK;
    }
  return err(ENOMEM_);
}
int cudaFree(void *p) {
  for (int k = 0; p && k < BLOCKS; k++)
    if (blocks[k].p == p) {
      used -= blocks[k].n;
      blocks[k].p = NULL;
      free(p);
      break;
    }
  return OK;
}
int cudaMalloc(void **p, size_t n) { return get(p, n); }
int cudaMallocAsync(void **p, size_t n, void *s) { (void)s; return get(p, n); }
int cudaFreeAsync(void *p, void *s) { (void)s; return cudaFree(p); }
int cudaMallocHost(void **p, size_t n) { return (*p = calloc(n ? n : 1, 1)) ? OK : err(ENOMEM_); }
int cudaHostAlloc(void **p, size_t n, unsigned f) { (void)f; return cudaMallocHost(p, n); }
int cudaFreeHost(void *p) { free(p); return OK; }
int cudaMemGetInfo(size_t *fr, size_t *total) { *fr = limit - used; *total = limit; return OK; }
int cudaMemcpy(void *d, const void *s, size_t n, int k) { (void)k; memcpy(d, s, n); return OK; }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int k, void *st) { (void)st; return cudaMemcpy(d, s, n, k); }
int cudaMemset(void *d, int v, size_t n) { memset(d, v, n); return OK; }
int cudaMemsetAsync(void *d, int v, size_t n, void *st) { (void)st; return cudaMemset(d, v, n); }
int cudaGetSymbolAddress(void **p, const void *s) { (void)s; return get(p, 1 << 23); }
int cudaDeviceGetDefaultMemPool(void **p, int d) { (void)d; *p = &used; return OK; }
int cudaMemPoolSetAttribute(void *p, int a, void *v) { (void)p; (void)a; (void)v; return OK; }

/* ---- device, streams, events, graphs */
int cudaGetDeviceCount(int *n) { *n = 1; return OK; }
int cudaGetDevice(int *d) { *d = 0; return OK; }
int cudaSetDevice(int d) { (void)d; return OK; }
int cudaDeviceGetAttribute(int *v, int a, int d) { (void)a; (void)d; *v = 148; return OK; }
int cudaDeviceSynchronize(void) { return OK; }
int cudaDeviceGetStreamPriorityRange(int *lo, int *hi) { *lo = 0; *hi = -5; return OK; }
int cudaStreamCreateWithPriority(void **s, unsigned f, int p) { (void)f; (void)p; *s = malloc(1); return OK; }
int cudaStreamCreateWithFlags(void **s, unsigned f) { return cudaStreamCreateWithPriority(s, f, 0); }
int cudaStreamDestroy(void *s) { free(s); return OK; }
int cudaStreamSynchronize(void *s) { (void)s; return OK; }
int cudaStreamWaitEvent(void *s, void *e, unsigned f) { (void)s; (void)e; (void)f; return OK; }
int cudaStreamBeginCapture(void *s, int m) { (void)s; (void)m; capturing = 1; return OK; }
int cudaStreamEndCapture(void *s, void **g) { (void)s; capturing = 0; *g = malloc(1); return OK; }
int cudaGraphInstantiate(void **x, void *g, unsigned long long f) {
  (void)g; (void)f;
  *x = malloc(1);
  instantiated++;
  return OK;
}
int cudaGraphLaunch(void *x, void *s) {
  (void)x; (void)s;
  if (fail_graph_launch) return err(ENOMEM_);
  graph_launches++;
  return OK;
}
int cudaGraphDestroy(void *g) { free(g); return OK; }
int cudaGraphExecDestroy(void *g) { free(g); return OK; }
int cudaEventCreate(void **e) { *e = malloc(1); return OK; }
int cudaEventCreateWithFlags(void **e, unsigned f) { (void)f; return cudaEventCreate(e); }
int cudaEventDestroy(void *e) { free(e); return OK; }
int cudaEventRecord(void *e, void *s) { (void)e; (void)s; return OK; }
int cudaEventSynchronize(void *e) { (void)e; return OK; }
int cudaEventElapsedTime(float *ms, void *a, void *b) { (void)a; (void)b; *ms = 1.f; return OK; }
int cudaGetLastError(void) { int e = last_error; last_error = 0; return e; }
const char *cudaGetErrorString(int e) { return e == ENOMEM_ ? "out of memory" : "fake error"; }
