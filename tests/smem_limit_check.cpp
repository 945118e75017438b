// allow_smem against a stand-in for the CUDA runtime with two devices: the
// limit belongs to (kernel, device), is set before the first launch there and
// once, also by threads that arrive together.
#include <atomic>
#include <cstdio>
#include <map>
#include <thread>
#include <vector>

#include "smem_limit.h"

static thread_local int t_device = 0;
static std::mutex g_mu;
static std::map<std::pair<int, const void*>, std::vector<int>> g_set;
static bool g_fail = false;

extern "C" cudaError_t cudaGetDevice(int* d) {
  *d = t_device;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaErrorInvalidValue;
  if (g_fail) return cudaErrorInvalidValue;
  std::lock_guard<std::mutex> lock(g_mu);
  g_set[{t_device, f}].push_back(v);
  return cudaSuccess;
}
extern "C" const char* cudaGetErrorString(cudaError_t) { return "stand-in"; }

static int a, b;
#define CHECK(x)                                     \
  if (!(x)) {                                        \
    std::printf("line %d: %s\n", __LINE__, #x);      \
    return 1;                                        \
  }

int main() {
  g_fail = true;  // a refusal is an error, and is not remembered
  try {
    drg::allow_smem(&a, 60000);
    CHECK(false);
  } catch (const drg::Error& e) {
    CHECK(e.code == DRG_ERR_CUDA);
  }
  g_fail = false;
  std::vector<std::thread> ts;
  std::atomic<int> missing{0};
  for (int k = 0; k < 16; ++k)
    ts.emplace_back([&, k] {
      t_device = k % 2;
      for (int i = 0; i < 1000; ++i) {
        const void* f = i % 2 ? &a : &b;
        drg::allow_smem(f, i % 2 ? 60000 : 100000);
        std::lock_guard<std::mutex> lock(g_mu);
        if (!g_set.count({t_device, f})) ++missing;  // a launch here would be refused
      }
    });
  for (auto& t : ts) t.join();
  CHECK(missing == 0);
  CHECK(g_set.size() == 4);
  for (auto& [k, v] : g_set) CHECK(v.size() == 1 && v[0] == (k.second == &a ? 60000 : 100000));
  std::printf("ok\n");
  return 0;
}
