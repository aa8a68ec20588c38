// HostPipe and HostCopy on a stand-in for the CUDA runtime: a call that fails while its
// upload is under way must leave no copy to be enqueued behind its final wait.
// Prints "<status> <copies enqueued> <of them after the stream's wait> <after finish>
// <every byte arrived> <error left for the next launch's check>".
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>

#include "../../stream-k-gemm_b200/csrc/skg_hostcopy.cu"

static std::atomic<int> g_copies{0}, g_late{0};
static std::atomic<bool> g_waited{false};
static bool g_no_pinned = false, g_registered = false;
static cudaError_t g_last = cudaSuccess;

extern "C" {
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  a->type = g_registered ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = g_no_pinned ? nullptr : malloc(n);
  return *p ? cudaSuccess : (g_last = cudaErrorMemoryAllocation);
}
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free((void*)e); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)malloc(1); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { g_waited = true; return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h,
                              cudaMemcpyKind, cudaStream_t) {
  std::this_thread::sleep_for(std::chrono::milliseconds(2));
  for (size_t r = 0; r < h; ++r) memcpy((char*)d + r * dp, (const char*)s + r * sp, w);
  ++g_copies;
  if (g_waited) ++g_late;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t t) {
  return cudaMemcpy2DAsync(d, n, s, n, n, 1, k, t);
}
}

namespace skg {
int fail(int code, const std::string&) { return code; }
int cuda_fail(cudaError_t, const char*) { return SKGEMM_ERR_CUDA; }
int consume_device_error(StreamWorkspace*, cudaStream_t) { return SKGEMM_OK; }
}  // namespace skg

int main(int argc, char** argv) {
  using namespace skg;
  const bool failing = argc > 1 && !strcmp(argv[1], "fail");
  g_no_pinned = argc > 1 && !strcmp(argv[1], "unpinned");
  g_registered = argc > 1 && !strcmp(argv[1], "pinned");
  const int chunks = 8;
  const size_t n = 4 << 20;
  std::vector<char> src(chunks * n), dst(chunks * n);
  for (size_t i = 0; i < src.size(); ++i) src[i] = (char)(i * 31 >> 7);
  DeviceState dev;
  dev.device = 0;
  HostPipe hp;
  int st = hp.init(&dev, chunks);
  HostCopy& up = hp.upload();
  for (int c = 0; c < chunks; ++c) up.add(c, dst.data() + c * n, n, src.data() + c * n, n, n, 1);
  st = up.start();
  for (int c = 0; c < chunks && !st; ++c) {
    st = up.wait_group(c);
    if ((g_registered || g_no_pinned) && g_copies != c + 1) st = SKGEMM_ERR_CUDA;  // later chunks' too
    if (failing && c == 1) st = SKGEMM_ERR_OOM;  // the chunk's launch failed
  }
  const int got = hp.finish(st);
  const int seen = g_copies;
  std::this_thread::sleep_for(std::chrono::milliseconds(60));
  printf("%d %d %d %d %d %d\n", got, seen, (int)g_late, (int)g_copies - seen, src == dst ? 1 : 0,
         (int)g_last);
  return 0;
}
