// The serving scheduler against an executor whose requests complete with a device
// error word: run on the host, no GPU. Prints "<status> <requests run> <message>".
#include "../../stream-k-gemm_b200/csrc/skg_serve.cu"

namespace skg {
static std::string g_msg;
int fail(int code, const std::string& m) {
  g_msg = m;
  return code;
}
int cuda_fail(cudaError_t, const char* what) { return fail(SKGEMM_ERR_CUDA, what); }
std::string device_error_text(uint32_t w) { return "word " + std::to_string(w); }
// Never reached by the scheduler.
DeviceState* current_device(int* st) { *st = SKGEMM_ERR_NO_DEVICE; return nullptr; }
StreamWorkspace* stream_workspace(DeviceState*, cudaStream_t, size_t, int*, size_t) { return nullptr; }
int launch_band_to_grid(int64_t, int64_t, const double*, double*, cudaStream_t) { return 0; }
Fp64Problem gemm_packed_problem(int64_t, int64_t, int64_t, const double*, const double*, double*,
                                int64_t, double, double) { return {}; }
Fp64Problem syrk_problem(int64_t, int64_t, const double*, double*, int64_t, double, double) { return {}; }
Fp64Problem rot_problem(int64_t, int64_t, const double*, const double*, double*, bool) { return {}; }
GroupRing* group_ring_create(DeviceState*, int) { return nullptr; }
void group_ring_destroy(GroupRing*) {}
int group_ring_reserve(GroupRing*, int) { return 0; }
int group_ring_submit(GroupRing*, const std::vector<Fp64Problem>&, cudaStream_t, int*, const uint32_t**) { return 0; }
int group_ring_error(GroupRing*) { return 0; }
size_t group_ring_bytes(const GroupRing*) { return 0; }
int ozaki_reserve(DeviceState*, cudaStream_t, int64_t, int64_t, int) { return 0; }
size_t ozaki_stream_bytes(DeviceState*, cudaStream_t) { return 0; }
}  // namespace skg
int skgemm_dsubspace_packed_dev(int64_t, int64_t, const double*, const double*, double*, int64_t, double*,
                                int64_t, skgemm_options_t*, void*) { return 0; }
int skgemm_drot_dev_opt(int64_t, int64_t, const double*, const double*, double*, skgemm_options_t*, void*) { return 0; }
int skgemm_stream_status(void*) { return 0; }
int skgemm_stream_release(void*) { return 0; }

namespace skg { namespace serve {
struct FailingExec : SimExec {
  int bad = -1, ran = 0;
  uint32_t req_word(Req& r) override { return r.idx == bad ? 0x201u : 0u; }
  uint32_t batch_word(Batch& b) override {
    for (int i : b.s2)
      if (i == bad) return 0x101u;
    return 0u;
  }
  int finish(Req&, const skgemm_serve_request_t&) override { ++ran; return SKGEMM_OK; }
};
}}  // namespace skg::serve

int main(int argc, char** argv) {
  using namespace skg::serve;
  const bool native = argc > 1 && argv[1][0] == 'n';
  const int bad = argc > 2 ? atoi(argv[2]) : -1;
  const int n = 6;
  skgemm_serve_request_t io[n] = {};
  for (int i = 0; i < n; ++i) {
    io[i].Ng = 1600 + 16 * i;
    io[i].nb = 32;
  }
  skgemm_serve_options_t o = {};
  o.precision = native ? SKGEMM_PREC_NATIVE : SKGEMM_PREC_OZAKI_I8;
  o.max_inflight = 1;
  FailingExec ex;
  ex.bad = bad;
  Arena arena((size_t)1 << 32);
  const int st = schedule(io, n, o, ex, arena, native ? 0 : 1);
  printf("%d %d %s\n", st, ex.ran, skg::g_msg.c_str());
  return 0;
}
