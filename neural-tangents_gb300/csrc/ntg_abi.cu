// Library-level plumbing of the C ABI: per-thread error messages, version,
// and the launch counter reported by ntg_launch_count().
#include <cstdio>
#include <mutex>
#include <string>

#include "ntg_common.cuh"

namespace ntg {

static thread_local std::string g_last_error;
static std::atomic<uint64_t> g_launches{0};

void set_error(const std::string& msg) { g_last_error = msg; }

int fail(int code, const std::string& msg) {
  g_last_error = msg;
  return code;
}

int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    return fail(NTG_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
  }
  return NTG_OK;
}

void note_launch(uint64_t n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

constexpr int kMaxDevices = 64;

int* device_error_word() {
  static std::once_flag once;
  static int* words = nullptr;
  std::call_once(once, [] {
    // the first launch of a process may be under stream capture, which allows this
    // allocation (no stream is involved) in the relaxed mode only
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    void* p = nullptr;
    if (cudaHostAlloc(&p, kMaxDevices * sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped) ==
        cudaSuccess) {
      words = static_cast<int*>(p);
      for (int i = 0; i < kMaxDevices; ++i) words[i] = 0;
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
  });
  int dev = 0;
  if (!words || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
    return nullptr;
  return words + dev;  // unified addressing: the same address on the device
}

static std::atomic<int32_t> g_tune[NTG_TUNE_COUNT] = {{4}};

int32_t tune(int32_t knob) { return g_tune[knob].load(std::memory_order_relaxed); }

}  // namespace ntg

extern "C" const char* ntg_last_error(void) { return ntg::g_last_error.c_str(); }

extern "C" const char* ntg_version(void) { return "nt_gb300 0.1.0 (sm_103a)"; }

extern "C" uint64_t ntg_launch_count(void) {
  return ntg::g_launches.load(std::memory_order_relaxed);
}

extern "C" int ntg_tune_set(int32_t knob, int32_t value) {
  if (knob == NTG_TUNE_STENCIL_RING) {
    if (value != 2 && value != 3 && value != 4 && value != 6)
      return ntg::fail(NTG_ERR_INVALID_ARG, "ntg_tune_set: stencil ring must be 2, 3, 4 or 6");
  } else {
    return ntg::fail(NTG_ERR_INVALID_ARG, "ntg_tune_set: unknown knob");
  }
  ntg::g_tune[knob].store(value, std::memory_order_relaxed);
  return NTG_OK;
}

extern "C" int32_t ntg_tune_get(int32_t knob) {
  if (knob < 0 || knob >= NTG_TUNE_COUNT) return -1;
  return ntg::tune(knob);
}

extern "C" int ntg_device_status(void) {
  int* word = ntg::device_error_word();
  if (!word) return ntg::fail(NTG_ERR_CUDA, "ntg_device_status: no device error word");
  // what the legacy stream and the streams that block on it still run may set the word
  if (cudaStreamSynchronize(nullptr) != cudaSuccess)
    return ntg::check_launch("ntg_device_status");
  const int v = __atomic_exchange_n(word, 0, __ATOMIC_ACQ_REL);
  if (v != 0) return ntg::fail(v, "a bounded device wait ran out in a streamed kernel");
  return NTG_OK;
}
