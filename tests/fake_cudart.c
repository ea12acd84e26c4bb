/* CUDA runtime calls that fail on request: preloaded in front of libcudart by a test's child process, which sets the
 * counters. The failing call never reaches the runtime. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>

typedef struct { unsigned x, y, z; } fake_dim3;

int fail_cudaMalloc = 0, fail_cudaLaunchCooperativeKernel = 0; /* how many of the next calls fail */
int code_cudaLaunchCooperativeKernel = 0;                      /* with this error */

static void* real(const char* name) {
  static void* lib;
  if (!lib) lib = dlopen("libcudart.so.13", RTLD_NOW | RTLD_GLOBAL);
  return dlsym(lib, name);
}

int cudaMalloc(void** p, size_t n) {
  if (fail_cudaMalloc > 0) {
    --fail_cudaMalloc;
    return 2; /* cudaErrorMemoryAllocation */
  }
  return ((int (*)(void**, size_t))real("cudaMalloc"))(p, n);
}

int cudaLaunchCooperativeKernel(const void* f, fake_dim3 grid, fake_dim3 block, void** args, size_t smem, void* st) {
  if (fail_cudaLaunchCooperativeKernel > 0) {
    --fail_cudaLaunchCooperativeKernel;
    return code_cudaLaunchCooperativeKernel;
  }
  return ((int (*)(const void*, fake_dim3, fake_dim3, void**, size_t, void*))real("cudaLaunchCooperativeKernel"))(
      f, grid, block, args, smem, st);
}
