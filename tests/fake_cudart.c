/* A CUDA runtime without a device, for tests of the library's host code on
 * the CPU (tests/fake_cuda.py links the library's own objects against it):
 * device memory is host memory, copies are done at once, kernels do nothing
 * but are counted, and any call can be made to fail.  Copies and kernels
 * count as in flight until the host waits for their stream, for a stream that
 * waits for them, or for the device. */
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

#define MAXK 512
static struct {
  const void *fn;
  const char *name;
} kern[MAXK];
static int n_kern, n_launch, fail_in;
/* streams: what is in flight, and the streams that each waits for */
#define MAXS 256
static struct CUstream_st {
  int pending, n_dep;
  cudaStream_t dep[64];
} streams[MAXS];
static int n_streams = 1; /* 0: the default stream */
struct CUevent_st {
  cudaStream_t s;
};
static char log_[1 << 16];
static char fail_name[64];
static cudaError_t last;
static float elapsed_ms = 1.f;
static float (*elapsed_cb)(void);
static void (*launch_cb)(const char *, void **);

/* ---- the tests' side ---- */
static void sync_all(void)
{
  for (int i = 0; i < n_streams; i++) streams[i].pending = streams[i].n_dep = 0;
}
void fake_reset(void)
{
  sync_all();
  n_launch = fail_in = 0;
  log_[0] = 0;
  last = cudaSuccess;
}
/* the nth call of the named function from now on fails, once */
void fake_fail(const char *name, int nth)
{
  strncpy(fail_name, name, sizeof(fail_name) - 1);
  fail_in = nth;
}
int fake_launches(void) { return n_launch; }
/* on every stream but one, and those that it waits for (NULL: on all) */
int fake_inflight(cudaStream_t but)
{
  int n = 0, skip[MAXS] = {0};
  if (but) skip[but - streams] = 1;
  for (int round = 0; round < n_streams; round++)
    for (int i = 0; i < n_streams; i++)
      for (int k = 0; skip[i] && k < streams[i].n_dep; k++) skip[streams[i].dep[k] - streams] = 1;
  for (int i = 0; i < n_streams; i++) n += skip[i] ? 0 : streams[i].pending;
  return n;
}
const char *fake_log(void) { return log_; } /* the launched kernels' names, a line each */
void fake_elapsed(float (*cb)(void)) { elapsed_cb = cb; }
/* stands in for the kernels: called with each launch's kernel name and arguments */
void fake_on_launch(void (*cb)(const char *, void **)) { launch_cb = cb; }

static void enqueue(cudaStream_t s) { (s ? s : streams)->pending++; }
static void finish(cudaStream_t s)
{
  const int n = s->n_dep;
  s->pending = s->n_dep = 0;
  for (int i = 0; i < n; i++) finish(s->dep[i]);
}
static int fails(const char *name)
{
  if (!fail_in || strcmp(name, fail_name) || --fail_in) return 0;
  last = cudaErrorMemoryAllocation;
  return 1;
}
#define FAIL() \
  if (fails(__func__)) return last

/* ---- registration and launch ---- */
typedef struct {
  unsigned x, y, z;
} D3;
static D3 cfg_g, cfg_b;
static size_t cfg_s;
static void *cfg_st;
unsigned __cudaPushCallConfiguration(D3 g, D3 b, size_t s, void *st)
{
  cfg_g = g;
  cfg_b = b;
  cfg_s = s;
  cfg_st = st;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(D3 *g, D3 *b, size_t *s, void **st)
{
  *g = cfg_g;
  *b = cfg_b;
  *s = cfg_s;
  *st = cfg_st;
  return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *f) { return (void **)f; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterFunction(void **h, const char *fn, char *dev, const char *name, int tl, void *t, void *b, void *bd,
                            void *gd, int *ws)
{
  if (n_kern < MAXK) {
    kern[n_kern].fn = fn;
    kern[n_kern++].name = name;
  }
}
void __cudaRegisterVar(void **h, char *var, char *addr, const char *name, int ext, size_t size, int c, int g) {}
cudaError_t cudaLaunchKernel(const void *fn, dim3 g, dim3 b, void **args, size_t s, cudaStream_t st)
{
  FAIL();
  n_launch++;
  enqueue(st);
  for (int i = 0; launch_cb && i < n_kern; i++)
    if (kern[i].fn == fn) launch_cb(kern[i].name, args);
  for (int i = 0; i < n_kern; i++)
    if (kern[i].fn == fn && strlen(log_) + strlen(kern[i].name) + 2 < sizeof(log_)) {
      strcat(log_, kern[i].name);
      strcat(log_, "\n");
    }
  return cudaSuccess;
}

/* ---- memory ---- */
cudaError_t cudaMalloc(void **p, size_t n)
{
  *p = NULL;
  FAIL();
  *p = calloc(1, n ? n : 1);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void *p)
{
  if (p) sync_all();
  free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned f) { return *p = calloc(1, n ? n : 1), cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned f) { return *d = h, cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { return *f = *t = (size_t)64 << 20, cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k)
{
  FAIL();
  memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st)
{
  FAIL();
  memmove(d, s, n);
  enqueue(st);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { return memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) { return memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemcpyToSymbolAsync(const void *s, const void *p, size_t n, size_t o, enum cudaMemcpyKind k,
                                    cudaStream_t st)
{
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *s) { return *p = (void *)s, cudaSuccess; }

/* ---- device, streams, events ---- */
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) { return *v = 148, cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int *lo, int *hi) { return *lo = 0, *hi = -1, cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v)
{
  FAIL();
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *f, int t, size_t s)
{
  return *n = 1, cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f)
{
  if (n_streams == MAXS) return cudaErrorMemoryAllocation;
  *s = &streams[n_streams++];
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned f, int p) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
  finish(s ? s : streams);
  FAIL();
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f)
{
  FAIL();
  if (e->s && e->s != s && s->n_dep < 64) s->dep[s->n_dep++] = e->s;
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = calloc(1, sizeof(**e)), cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
  FAIL();
  return e->s = s ? s : streams, cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b)
{
  return *ms = elapsed_cb ? elapsed_cb() : elapsed_ms, cudaSuccess;
}
cudaError_t cudaGetLastError(void)
{
  FAIL();
  cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t e) { return "failed by the test"; }
