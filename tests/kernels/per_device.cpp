// csrc/per_device.cuh on the host alone: the two CUDA calls that it makes are defined here and count.
#include "per_device.cuh"

static int device = 0, calls = 0;
static bool fail = false;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) {
  ++calls;
  return fail ? cudaErrorInvalidValue : cudaSuccess;
}

static void one() {}
static void two() {}

// Asks for kernel 1 or 2 on `on`; returns the status and, in the next call of taken(), the attribute calls so far.
extern "C" int ask(int kernel, int on, int failing) {
  device = on;
  fail = failing != 0;
  return kernel == 1 ? (int)tl_allow_smem<one>(1000) : (int)tl_allow_smem<two>(1000);
}
extern "C" int taken() { return calls; }
