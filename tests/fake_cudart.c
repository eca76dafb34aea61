/* Stands in front of libcudart (LD_PRELOAD): makes chosen calls fail, or a
 * device appear, so that the library's host code is tested without them.
 * FAKE_SMS=n: a device of n multiprocessors where there is none.
 * FAKE_REFUSE=1: no cooperative and no cluster launch is accepted. */
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <stdlib.h>
#include <string.h>

static int refuse(void) { return getenv("FAKE_REFUSE") != NULL; }
static int sms(void) { return getenv("FAKE_SMS") ? atoi(getenv("FAKE_SMS")) : 0; }
/* the runtime that the library has loaded, which is not in the global scope */
static void* real(const char* name) {
  static void* rt;
  if (!rt) rt = dlopen("libcudart.so.13", RTLD_LAZY);
  return dlsym(rt, name);
}
#define REAL(name) ((__typeof__(&name))real(#name))

cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 g, dim3 b, void** a, size_t s, cudaStream_t st) {
  return refuse() ? cudaErrorCooperativeLaunchTooLarge : REAL(cudaLaunchCooperativeKernel)(f, g, b, a, s, st);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a) {
  return refuse() ? cudaErrorLaunchOutOfResources : REAL(cudaLaunchKernelExC)(c, f, a);
}
cudaError_t cudaGetDevice(int* d) {
  if (!sms()) return REAL(cudaGetDevice)(d);
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp* p, int d) {
  if (!sms()) return REAL(cudaGetDeviceProperties)(p, d);
  memset(p, 0, sizeof *p);
  p->multiProcessorCount = sms();
  p->sharedMemPerBlockOptin = 232448;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
  return sms() ? cudaSuccess : REAL(cudaFuncSetAttribute)(f, a, v);
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int b, size_t s, unsigned fl) {
  if (!sms()) return REAL(cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags)(n, f, b, s, fl);
  *n = 1;
  return cudaSuccess;
}
