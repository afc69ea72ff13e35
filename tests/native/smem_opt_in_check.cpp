// smem_opt_in against a fake CUDA runtime: the attribute is set once on every device that a kernel is launched on, and a
// device on which setting it failed is tried again. Built and run by tests/test_dispatch_cpu.py.
#include <string>

#include "host_util.h"

static int g_dev = 0;
static cudaError_t g_result = cudaSuccess;
static std::string g_log;

extern "C" {
cudaError_t CUDARTAPI cudaGetDevice(int* d) {
  *d = g_dev;
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaFuncSetAttribute(const void*, enum cudaFuncAttribute a, int bytes) {
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaErrorInvalidValue;
  g_log += std::to_string(g_dev) + ":" + std::to_string(bytes) + (g_result == cudaSuccess ? " " : "! ");
  return g_result;
}
const char* CUDARTAPI cudaGetErrorString(cudaError_t) { return "fake"; }
}

static void kernel_a(int) {}
static void kernel_b(int) {}

static int launch(int dev, bool a) {
  static std::atomic<uint64_t> in_a{0}, in_b{0};
  g_dev = dev;
  return a ? tb::smem_opt_in(in_a, kernel_a, 100) : tb::smem_opt_in(in_b, kernel_b, 200);
}

int main() {
  int bad = 0;
  bad |= launch(0, true) | launch(0, true) | launch(1, true) | launch(0, true) | launch(1, true);
  bad |= launch(1, false) | launch(63, false) | launch(63, false);
  g_result = cudaErrorInvalidValue;
  bad |= launch(2, true) == 0;
  g_result = cudaSuccess;
  bad |= launch(2, true) | launch(2, true);
  bad |= launch(64, true) | launch(64, true);   // beyond the set: every time
  puts(g_log.c_str());
  return bad;
}
