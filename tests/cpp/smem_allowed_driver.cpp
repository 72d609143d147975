// smem_allowed.h against a fake runtime: which device the attribute was set on.
#include "smem_allowed.h"

#include <cstdio>
#include <utility>
#include <vector>

static int g_device = 0, g_fail = 0;
static std::vector<std::pair<int, int>> g_set;  // (device, bytes)

extern "C" cudaError_t cudaGetDevice(int* device) {
  *device = g_device;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int value) {
  if (g_fail) return cudaErrorInvalidValue;
  g_set.push_back({g_device, value});
  return cudaSuccess;
}

int main() {
  gprx::SmemAllowed allowed;
  bool failed = false, ok = true;
  const int devices[] = {0, 0, 1, 1, 0, 3, 70, 70};
  for (int d : devices) {
    g_device = d;
    if (d == 3) {  // a refusal is reported and asked again
      g_fail = 1;
      failed = allowed(nullptr, 1000) == cudaErrorInvalidValue;
      g_fail = 0;
    }
    ok = ok && allowed(nullptr, 1000) == cudaSuccess;
  }
  std::printf("{\"ok\": %d, \"failed\": %d, \"set\": [", ok, failed);
  for (size_t i = 0; i < g_set.size(); ++i) std::printf("%s%d", i ? ", " : "", g_set[i].first);
  std::printf("]}\n");
}
