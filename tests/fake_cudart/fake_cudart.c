/* A CUDA runtime for tests of the library's host side without a GPU: loaded before libcudart
 * (LD_PRELOAD), it serves "device" and pinned memory from the heap, accepts every launch
 * without running it, and counts the allocations. */
#include <stdlib.h>
#include <string.h>

int fake_allocs = 0;              /* cudaMalloc and cudaMallocHost calls so far */
size_t fake_sizes[4096];          /* their sizes in bytes */
int fake_fail = 0;                /* the fake_fail-th call from now on fails */

static int take(void **p, size_t n) {
  if (fake_fail && --fake_fail == 0) return 2;   /* cudaErrorMemoryAllocation */
  if (fake_allocs < 4096) fake_sizes[fake_allocs] = n;
  ++fake_allocs;
  *p = calloc(1, n ? n : 1);
  return *p ? 0 : 2;
}
int cudaMalloc(void **p, size_t n) { return take(p, n); }
int cudaMallocHost(void **p, size_t n) { return take(p, n); }
int cudaFree(void *p) { free(p); return 0; }
int cudaFreeHost(void *p) { free(p); return 0; }
int cudaMemcpy(void *d, const void *s, size_t n, int k) { (void)k; memcpy(d, s, n); return 0; }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int k, void *st) {
  (void)k; (void)st; memcpy(d, s, n); return 0;
}
int cudaMemsetAsync(void *d, int v, size_t n, void *st) { (void)st; memset(d, v, n); return 0; }
int cudaSetDevice(int d) { (void)d; return 0; }
int cudaGetDevice(int *d) { *d = 0; return 0; }
int cudaGetDeviceCount(int *n) { *n = 1; return 0; }
int cudaDeviceSynchronize(void) { return 0; }
int cudaDeviceGetAttribute(int *v, int a, int d) { (void)a; (void)d; *v = 148; return 0; }
int cudaStreamSynchronize(void *s) { (void)s; return 0; }
int cudaFuncSetAttribute(const void *f, int a, int v) { (void)f; (void)a; (void)v; return 0; }
int fake_launch_fail = 0;         /* the fake_launch_fail-th launch from now on fails */
int fake_last = 0;                /* the error that cudaGetLastError reports and forgets */
static int launch(void) {
  if (fake_launch_fail && --fake_launch_fail == 0) return fake_last = 1;   /* cudaErrorInvalidValue */
  return 0;
}
int cudaGetLastError(void) { const int e = fake_last; fake_last = 0; return e; }
int cudaPeekAtLastError(void) { return fake_last; }
int cudaLaunchKernelExC(const void *c, const void *f, void **a) { (void)c; (void)f; (void)a; return launch(); }
struct fake_dim3 { unsigned x, y, z; };
int cudaLaunchKernel(const void *f, struct fake_dim3 g, struct fake_dim3 b, void **a, size_t m, void *s) {
  (void)f; (void)g; (void)b; (void)a; (void)m; (void)s; return launch();
}
int cudaStreamCreateWithFlags(void **s, unsigned f) { (void)f; *s = malloc(1); return *s ? 0 : 2; }
int cudaStreamDestroy(void *s) { free(s); return 0; }
int cudaStreamWaitEvent(void *s, void *e, unsigned f) { (void)s; (void)e; (void)f; return 0; }
int cudaEventCreateWithFlags(void **e, unsigned f) { (void)f; *e = malloc(1); return *e ? 0 : 2; }
int cudaEventDestroy(void *e) { free(e); return 0; }
int cudaEventRecord(void *e, void *s) { (void)e; (void)s; return 0; }
int cudaEventSynchronize(void *e) { (void)e; return 0; }
