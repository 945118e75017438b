// ForkGuard against a stand-in for cudaStreamSynchronize: a call that fails
// after a fork waits for every forked stream before its buffers are freed; a
// joined one waits for none.
#include <cstdint>
#include <cstdio>
#include <stdexcept>
#include <string>

#include "stream_fork.h"

static std::string g_log;
extern "C" cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  g_log += "w" + std::to_string((intptr_t)s);
  return cudaSuccess;
}
struct Buffer {
  ~Buffer() { g_log += "f"; }
};

static void call(int fail_at) {
  Buffer buffer;
  drg::ForkGuard forked;
  for (int k = 1; k <= 3; ++k) {
    forked.add((cudaStream_t)(intptr_t)k);
    if (k == fail_at) throw std::runtime_error("launch");
  }
  forked.joined();
  if (fail_at == 4) throw std::runtime_error("after the join");
}
static std::string run(int fail_at) {
  g_log.clear();
  try {
    call(fail_at);
  } catch (const std::runtime_error&) {
    g_log += "e";
  }
  return g_log;
}

int main() {
  const char* expect[] = {"f", "w1fe", "w1w2fe", "w1w2w3fe", "fe"};
  for (int k = 0; k < 5; ++k)
    if (run(k) != expect[k]) {
      std::printf("%d: %s\n", k, g_log.c_str());
      return 1;
    }
  std::printf("ok\n");
  return 0;
}
