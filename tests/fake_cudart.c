/* A CUDA runtime that owns no GPU, for tests of the library's host side: memory is
 * host memory, copies and fills happen at once, kernels do not run (but for the
 * mirror of the control blocks, which the host waits for) and are only noted, and
 * a chosen launch, fill or copy is refused with an error code. */
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

typedef int err_t;
typedef struct { unsigned x, y, z; } dim3_t;
typedef struct { dim3_t grid, block; size_t smem; void* stream; void* attrs; unsigned n_attrs; } config_t;

static struct { const void* fn; const char* name; } g_kernel[1024];
static int g_kernels;
static char g_log[1 << 16], g_refuse[128];
static int g_refuse_fill, g_last, g_pool_live;

void fake_refuse(const char* part) { snprintf(g_refuse, sizeof g_refuse, "%s", part); }
void fake_refuse_fill(int on) { g_refuse_fill = on; }
int fake_pool_blocks(void) { return g_pool_live; }
const char* fake_log(void) { return g_log; }
void fake_clear_log(void) { g_log[0] = 0; }

static err_t ret(err_t e) { return e ? (g_last = e) : 0; }
err_t cudaGetLastError(void) { err_t e = g_last; g_last = 0; return e; }
const char* cudaGetErrorString(err_t e) { return e == 701 ? "too many resources requested for launch (fake)" : "fake error"; }

static err_t launch(const void* fn, void** args) {
  const char* name = "?";
  for (int i = 0; i < g_kernels; ++i)
    if (g_kernel[i].fn == fn) name = g_kernel[i].name;
  if (g_refuse[0] && strstr(name, g_refuse)) return ret(701);
  if (strlen(g_log) + strlen(name) + 2 < sizeof g_log) { strcat(g_log, name); strcat(g_log, "\n"); }
  if (strstr(name, "k_mirror")) memcpy(*(void**)args[1], *(void**)args[0], 4 * (size_t)*(int*)args[2]);
  return 0;
}
err_t cudaLaunchKernel(const void* fn, dim3_t g, dim3_t b, void** args, size_t sm, void* st) {
  (void)g; (void)b; (void)sm; (void)st;
  return launch(fn, args);
}
err_t cudaLaunchKernelExC(const config_t* c, const void* fn, void** args) { (void)c; return launch(fn, args); }

static config_t g_call;
unsigned __cudaPushCallConfiguration(dim3_t g, dim3_t b, size_t sm, void* st) {
  g_call.grid = g; g_call.block = b; g_call.smem = sm; g_call.stream = st;
  return 0;
}
err_t __cudaPopCallConfiguration(dim3_t* g, dim3_t* b, size_t* sm, void* st) {
  *g = g_call.grid; *b = g_call.block; *sm = g_call.smem; *(void**)st = g_call.stream;
  return 0;
}
void** __cudaRegisterFatBinary(void* f) { (void)f; static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterVar(void** h, char* v, char* a, const char* n, int e, size_t s, int c, int g) {
  (void)h; (void)v; (void)a; (void)n; (void)e; (void)s; (void)c; (void)g;
}
void __cudaRegisterFunction(void** h, const char* fn, char* d, const char* name, int t, void* a, void* b, void* c,
                            void* e, int* w) {
  (void)h; (void)d; (void)t; (void)a; (void)b; (void)c; (void)e; (void)w;
  if (g_kernels < 1024) { g_kernel[g_kernels].fn = fn; g_kernel[g_kernels++].name = name; }
}

static err_t get(void** p, size_t n) { return ret((*p = calloc(1, n ? n : 1)) ? 0 : 2); }
err_t cudaMalloc(void** p, size_t n) { return get(p, n); }
err_t cudaHostAlloc(void** p, size_t n, unsigned f) { (void)f; return get(p, n); }
err_t cudaFree(void* p) { free(p); return 0; }
err_t cudaFreeHost(void* p) { free(p); return 0; }
err_t cudaMallocFromPoolAsync(void** p, size_t n, void* pool, void* st) { (void)pool; (void)st; ++g_pool_live; return get(p, n); }
err_t cudaFreeAsync(void* p, void* st) { (void)st; --g_pool_live; free(p); return 0; }
err_t cudaMemPoolCreate(void** p, const void* props) { (void)props; static int x; *p = &x; return 0; }
err_t cudaMemPoolSetAttribute(void* p, int a, void* v) { (void)p; (void)a; (void)v; return 0; }
err_t cudaMemcpy(void* d, const void* s, size_t n, int k) { (void)k; memcpy(d, s, n); return 0; }
err_t cudaMemcpyAsync(void* d, const void* s, size_t n, int k, void* st) { (void)k; (void)st; memcpy(d, s, n); return 0; }
err_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return 0; }
err_t cudaMemsetAsync(void* d, int v, size_t n, void* st) {
  (void)st;
  if (g_refuse_fill) return ret(1);
  memset(d, v, n);
  return 0;
}

err_t cudaGetDevice(int* d) { *d = 0; return 0; }
err_t cudaDeviceGetAttribute(int* v, int a, int d) { (void)a; (void)d; *v = 148; return 0; }
err_t cudaFuncSetAttribute(const void* f, int a, int v) { (void)f; (void)a; (void)v; return 0; }
err_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int b, size_t s, unsigned fl) {
  (void)f; (void)b; (void)s; (void)fl;
  *n = 2;
  return 0;
}
err_t cudaGetSymbolAddress(void** p, const void* s) { (void)s; static char buf[64]; *p = buf; return 0; }
err_t cudaEventCreate(void** e) { return get(e, 8); }
err_t cudaEventCreateWithFlags(void** e, unsigned f) { (void)f; return get(e, 8); }
err_t cudaEventDestroy(void* e) { free(e); return 0; }
err_t cudaEventRecord(void* e, void* st) { (void)e; (void)st; return 0; }
err_t cudaEventSynchronize(void* e) { (void)e; return 0; }
err_t cudaEventElapsedTime(float* ms, void* a, void* b) { (void)a; (void)b; *ms = 0.f; return 0; }
err_t cudaStreamCreateWithFlags(void** s, unsigned f) { (void)f; return get(s, 8); }
err_t cudaStreamSynchronize(void* s) { (void)s; return 0; }
err_t cudaStreamBeginCapture(void* s, int m) { (void)s; (void)m; return ret(801); }
err_t cudaStreamEndCapture(void* s, void** g) { (void)s; *g = 0; return ret(801); }
err_t cudaGraphDestroy(void* g) { (void)g; return 0; }
err_t cudaGraphExecDestroy(void* g) { (void)g; return 0; }
err_t cudaGraphInstantiate(void** x, void* g, unsigned long long f) { (void)x; (void)g; (void)f; return ret(801); }
err_t cudaGraphLaunch(void* x, void* s) { (void)x; (void)s; return ret(801); }
