// ds_smem.h against a fake of the two runtime calls: the opt-in is asked for on every
// device that a kernel runs on, once each, and again after a failure.
#include "../../diffsplat_b200/csrc/ds_smem.h"

#include <cstdio>

static int g_device = 0, g_calls = 0;
static cudaError_t g_answer = cudaSuccess;
extern "C" cudaError_t cudaGetDevice(int* dev) {
  *dev = g_device;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) {
  ++g_calls;
  return g_answer;
}

static void kernel() {}

#define CHECK(x) \
  if (!(x)) return std::printf("line %d: %s\n", __LINE__, #x), 1

int main() {
  std::atomic<uint64_t> done{0}, other{0};
  CHECK(ds::allow_smem(kernel, 48 * 1024, done) == cudaSuccess && g_calls == 0);
  for (int round = 0; round < 3; ++round)
    for (g_device = 0; g_device < 64; ++g_device)
      CHECK(ds::allow_smem(kernel, 200 * 1024, done) == cudaSuccess);
  CHECK(g_calls == 64);
  g_device = 70;  // past the mask: every time
  ds::allow_smem(kernel, 200 * 1024, done);
  ds::allow_smem(kernel, 200 * 1024, done);
  CHECK(g_calls == 66);
  g_device = 1;
  g_answer = cudaErrorInvalidValue;
  CHECK(ds::allow_smem(kernel, 200 * 1024, other) == cudaErrorInvalidValue && other.load() == 0);
  g_answer = cudaSuccess;
  CHECK(ds::allow_smem(kernel, 200 * 1024, other) == cudaSuccess && other.load() == 2);
  CHECK(g_calls == 68);
  std::puts("ok");
  return 0;
}
