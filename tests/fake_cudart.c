/* A CUDA runtime without a device, for tests of the library's host code: it is
 * preloaded in front of libcudart.  Device memory is lazily committed host
 * memory, kernels do nothing but are counted by name, and a test can make the
 * launches of a kernel fail or have it write one word.  k_read_back, which
 * brings values to the host, is carried out. */
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include <sys/mman.h>

#define MAXK 1024
static const void *k_fun[MAXK];
static const char *k_name[MAXK];
static long k_count[MAXK];
static int k_n;
static struct { char *p; size_t n; } blk[4096];
static int blk_n;
static cudaError_t last;
static char fail_name[64], poke_name[64];
static cudaError_t fail_err;
static int poke_arg, poke_ptr, poke_word;
static unsigned poke_val;
static char handle_storage[8];

/* launches of kernels whose (mangled) name contains `name` return err */
void fake_fail(const char *name, int err) { snprintf(fail_name, sizeof fail_name, "%s", name); fail_err = (cudaError_t)err; }
/* a launch of `name` writes val to word `word` of the memory that the pointer at byte `ptr` of argument `arg` points to */
void fake_poke(const char *name, int arg, int ptr, int word, unsigned val) {
    snprintf(poke_name, sizeof poke_name, "%s", name);
    poke_arg = arg; poke_ptr = ptr; poke_word = word; poke_val = val;
}
long fake_count(const char *name) {
    long c = 0;
    for (int i = 0; i < k_n; i++)
        if (strstr(k_name[i], name)) c += k_count[i];
    return c;
}
void fake_reset(void) { memset(k_count, 0, sizeof k_count); fail_name[0] = poke_name[0] = 0; last = cudaSuccess; }

/* ---- registration of kernels (called by the compiler's start-up code) */
void **__cudaRegisterFatBinary(void *f) { (void)f; return (void **)handle_storage; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterVar(void **h, char *v, char *a, const char *n, int e, size_t s, int c, int g) {
    (void)h; (void)v; (void)a; (void)n; (void)e; (void)s; (void)c; (void)g;
}
void __cudaRegisterFunction(void **h, const char *fun, char *dev, const char *name, int tl, void *a, void *b, void *c, void *d,
                            int *w) {
    (void)h; (void)dev; (void)tl; (void)a; (void)b; (void)c; (void)d; (void)w;
    if (k_n < MAXK) { k_fun[k_n] = fun; k_name[k_n++] = name; }
}

/* ---- launches */
struct rb_list { const unsigned char *src[8]; unsigned bytes[8], off[8]; int n; };
static cudaError_t set(cudaError_t e) { if (e) last = e; return e; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *cfg, const void *fun, void **args) {
    (void)cfg;
    for (int i = 0; i < k_n; i++) {
        if (k_fun[i] != fun) continue;
        if (fail_name[0] && strstr(k_name[i], fail_name)) return set(fail_err);
        k_count[i]++;
        if (poke_name[0] && strstr(k_name[i], poke_name))
            ((unsigned *)(*(char **)((char *)args[poke_arg] + poke_ptr)))[poke_word] = poke_val;
        if (strstr(k_name[i], "k_read_back")) {
            const struct rb_list *l = (const struct rb_list *)args[0];
            unsigned char *dst = *(unsigned char **)args[1];
            for (int j = 0; j < l->n; j++) memcpy(dst + l->off[j], l->src[j], l->bytes[j]);
        }
        return cudaSuccess;
    }
    return set(cudaErrorInvalidDeviceFunction);
}
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) { (void)f; (void)a; (void)v; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t e) { (void)e; return "fake"; }

/* ---- memory */
static cudaError_t get(void **p, size_t n) {
    void *q = mmap(NULL, n ? n : 1, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (q == MAP_FAILED || blk_n == 4096) return set(cudaErrorMemoryAllocation);
    blk[blk_n].p = q;
    blk[blk_n++].n = n;
    *p = q;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { return get(p, n); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned f) { (void)f; return get(p, n); }
cudaError_t cudaFree(void *p) { (void)p; return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { (void)p; return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned f) { (void)f; *d = h; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p) {
    memset(a, 0, sizeof *a);
    for (int i = 0; i < blk_n; i++)
        if ((char *)p >= blk[i].p && (char *)p < blk[i].p + blk[i].n) a->type = cudaMemoryTypeDevice;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
    (void)k; (void)st;
    if (n <= (16u << 20)) memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) { return cudaMemcpyAsync(d, s, n, k, 0); }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
    (void)st;
    if (n <= (16u << 20)) memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { return cudaMemsetAsync(d, v, n, 0); }

/* ---- device, streams, events */
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { (void)d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) { (void)a; (void)d; *v = 152; return cudaSuccess; }
cudaError_t cudaDeviceSetLimit(enum cudaLimit l, size_t v) { (void)l; (void)v; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = (cudaStream_t)handle_storage; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s; (void)e; (void)f; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)handle_storage; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void)f; return cudaEventCreate(e); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
