/* A CUDA runtime without a GPU, preloaded by the tests that name it: memory is
 * host memory, kernels do nothing, every allocation, launch, event call and
 * stream synchronisation is logged, and one event call can be made to fail. */
#include <stdlib.h>
#include <string.h>

typedef struct { unsigned x, y, z; } dim3_t;
typedef int err_t;

static struct { char op; long stream; } g_log[1 << 16];
static int g_n, g_left = -1, g_last;
static char g_op;
static long g_handles = 1;

static void note(char op, void* stream) {
  if (g_n < (1 << 16)) g_log[g_n].op = op, g_log[g_n].stream = (long)stream, g_n++;
}
static err_t call(char op, void* stream) {  /* 'R' record, 'W' wait */
  if (op == g_op && g_left >= 0 && g_left-- == 0) {
    note('F', stream);
    return g_last = 999;
  }
  note(op, stream);
  return 0;
}
/* the nth call of kind op from here on fails (nth < 0: none); the log restarts */
void fake_fail(char op, int nth) { g_op = op, g_left = nth, g_n = 0; }
int fake_log(char* ops, long* streams, int max) {
  for (int i = 0; i < g_n && i < max; i++) ops[i] = g_log[i].op, streams[i] = g_log[i].stream;
  return g_n;
}

err_t cudaMalloc(void** p, size_t n) { note('M', (void*)n); return (*p = calloc(n + 256, 1)) ? 0 : 2; }
err_t cudaFree(void* p) { free(p); return 0; }
err_t cudaMemcpy(void* d, const void* s, size_t n, int k) { memcpy(d, s, n); return 0; }
err_t cudaMemcpyAsync(void* d, const void* s, size_t n, int k, void* st) { memcpy(d, s, n); return 0; }
err_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return 0; }
err_t cudaMemsetAsync(void* d, int v, size_t n, void* st) { memset(d, v, n); return 0; }
err_t cudaSetDevice(int d) { return 0; }
err_t cudaGetDevice(int* d) { *d = 0; return 0; }
err_t cudaDeviceGetAttribute(int* v, int a, int d) { *v = 152; return 0; }
err_t cudaGetLastError(void) { int e = g_last; g_last = 0; return e; }
const char* cudaGetErrorString(err_t e) { return e ? "made to fail" : "no error"; }
err_t cudaStreamCreateWithFlags(void** s, unsigned f) { *s = (void*)(g_handles++ * 64); return 0; }
err_t cudaStreamDestroy(void* s) { return 0; }
err_t cudaStreamSynchronize(void* s) { note('S', s); return 0; }
err_t cudaStreamWaitEvent(void* s, void* e, unsigned f) { return call('W', s); }
err_t cudaEventCreate(void** e) { *e = (void*)(g_handles++ * 64); return 0; }
err_t cudaEventCreateWithFlags(void** e, unsigned f) { *e = (void*)(g_handles++ * 64); return 0; }
err_t cudaEventDestroy(void* e) { return 0; }
err_t cudaEventRecord(void* e, void* s) { return call('R', s); }
err_t cudaEventSynchronize(void* e) { return 0; }
err_t cudaEventElapsedTime(float* t, void* a, void* b) { *t = 0; return 0; }
err_t cudaFuncSetAttribute(const void* f, int a, int v) { return 0; }

static struct { dim3_t g, b; size_t sm; void* st; } g_cfg;
unsigned __cudaPushCallConfiguration(dim3_t g, dim3_t b, size_t sm, void* st) {
  g_cfg.g = g, g_cfg.b = b, g_cfg.sm = sm, g_cfg.st = st;
  return 0;
}
err_t __cudaPopCallConfiguration(dim3_t* g, dim3_t* b, size_t* sm, void* st) {
  *g = g_cfg.g, *b = g_cfg.b, *sm = g_cfg.sm, *(void**)st = g_cfg.st;
  return 0;
}
err_t __cudaGetKernel(void** k, const void* f) { *k = (void*)f; return 0; }
err_t __cudaLaunchKernel(void* k, dim3_t g, dim3_t b, void** a, size_t sm, void* st) { note('L', st); return 0; }
err_t cudaLaunchKernel(const void* k, dim3_t g, dim3_t b, void** a, size_t sm, void* st) { note('L', st); return 0; }
void** __cudaRegisterFatBinary(void* f) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void** h) {}
void __cudaUnregisterFatBinary(void** h) {}
void __cudaRegisterFunction(void** h, const char* f, char* d, const char* n, int l, void* t, void* b, void* bd, void* gd, int* w) {}
void __cudaRegisterVar(void** h, char* v, char* d, const char* n, int e, size_t s, int c, int g) {}
