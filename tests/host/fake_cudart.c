/* A CUDA runtime without a GPU, for tests of the library's host code: two devices whose
 * memory is host memory and whose kernels do nothing.  As on a GPU, a launch with more
 * than 48 KB of dynamic shared memory is refused unless the kernel was opted in on the
 * current device. */
#include <stddef.h>
#include <stdlib.h>
#include <string.h>

enum { kDevices = 2, kFuncs = 4096, kInvalidValue = 1, kMaxDynamicSharedMemorySize = 8 };
static int device, last_error;
static struct { const void *func; int bytes[kDevices]; } funcs[kFuncs];
static int n_funcs, n_launches;

static int *opted(const void *func) {
    for (int i = 0; i < n_funcs; ++i)
        if (funcs[i].func == func) return &funcs[i].bytes[device];
    funcs[n_funcs].func = func;
    return &funcs[n_funcs++].bytes[device];
}

int fake_launches(void) { return n_launches; }

/* (the first members of cudaLaunchConfig_t) */
struct config { unsigned grid[3], block[3]; size_t smem; };
int cudaLaunchKernelExC(const struct config *c, const void *func, void **args) {
    (void)args;
    if (c->smem > 48 * 1024 && (size_t)*opted(func) < c->smem) return last_error = kInvalidValue;
    ++n_launches;
    return 0;
}
int cudaFuncSetAttribute(const void *func, int attr, int value) {
    if (attr == kMaxDynamicSharedMemorySize) *opted(func) = value;
    return 0;
}
/* (not zero: the launch is skipped) */
unsigned __cudaPushCallConfiguration(void) { return 1; }
int __cudaPopCallConfiguration(void) { return 0; }
int __cudaLaunchKernel(void) { return 0; }
int __cudaGetKernel(void) { return 0; }
void **__cudaRegisterFatBinary(void *bin) { static void *handle; (void)bin; return &handle; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterFunction(void) {}
void __cudaRegisterVar(void) {}

int cudaGetDeviceCount(int *n) { *n = kDevices; return 0; }
int cudaSetDevice(int d) { device = d; return 0; }
int cudaGetDevice(int *d) { *d = device; return 0; }
int cudaDeviceGetAttribute(int *v, int attr, int d) { (void)attr; (void)d; *v = 152; return 0; }
int cudaGetLastError(void) { const int e = last_error; last_error = 0; return e; }
const char *cudaGetErrorString(int e) { return e == kInvalidValue ? "invalid argument" : "no error"; }

int cudaMalloc(void **p, size_t n) { *p = calloc(n ? n : 1, 1); return 0; }
int cudaFree(void *p) { free(p); return 0; }
int cudaMallocHost(void **p, size_t n) { return cudaMalloc(p, n); }
int cudaHostAlloc(void **p, size_t n, unsigned flags) { (void)flags; return cudaMalloc(p, n); }
int cudaFreeHost(void *p) { return cudaFree(p); }
int cudaHostGetDevicePointer(void **d, void *h, unsigned flags) { (void)flags; *d = h; return 0; }
int cudaMemcpy(void *d, const void *s, size_t n, int kind) { (void)kind; memcpy(d, s, n); return 0; }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int kind, void *st) { (void)kind; (void)st; memcpy(d, s, n); return 0; }
int cudaMemsetAsync(void *d, int v, size_t n, void *st) { (void)st; memset(d, v, n); return 0; }

int cudaStreamCreateWithFlags(void **s, unsigned flags) { (void)flags; *s = malloc(1); return 0; }
int cudaStreamDestroy(void *s) { free(s); return 0; }
int cudaStreamSynchronize(void *s) { (void)s; return 0; }
int cudaEventCreate(void **e) { *e = malloc(1); return 0; }
int cudaEventCreateWithFlags(void **e, unsigned flags) { (void)flags; return cudaEventCreate(e); }
int cudaEventDestroy(void *e) { free(e); return 0; }
int cudaEventRecord(void *e, void *s) { (void)e; (void)s; return 0; }
int cudaEventSynchronize(void *e) { (void)e; return 0; }
