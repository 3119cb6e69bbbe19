// Library-level entry points: version, status strings, device queries and the
// workspace status word.
#include <atomic>
#include <mutex>

#include "common.cuh"

namespace sg {

static std::atomic<unsigned long long> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

int device_info(DeviceInfo* out) {
  static std::mutex mu;
  static DeviceInfo cache[64];
  static bool valid[64] = {false};
  int dev = 0;
  SG_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return SPLIT_ERR_CUDA;
  std::lock_guard<std::mutex> lock(mu);
  if (!valid[dev]) {
    DeviceInfo d;
    d.device = dev;
    SG_CUDA_TRY(cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, dev));
    SG_CUDA_TRY(cudaDeviceGetAttribute(&d.max_smem_optin,
                                       cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    int major = 0;
    SG_CUDA_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
    if (major < 10) return SPLIT_ERR_UNSUPPORTED;
    cache[dev] = d;
    valid[dev] = true;
  }
  *out = cache[dev];
  return SPLIT_OK;
}

}  // namespace sg

using namespace sg;

extern "C" unsigned long long split_launch_count(void) {
  return g_launches.load(std::memory_order_relaxed);
}

extern "C" const char* split_version(void) { return "split_gb300 0.1.0 (sm_103a)"; }

extern "C" const char* split_status_string(int status) {
  switch (status) {
    case SPLIT_OK: return "ok";
    case SPLIT_ERR_INVALID: return "invalid argument";
    case SPLIT_ERR_WORKSPACE: return "workspace too small or misaligned";
    case SPLIT_ERR_NOT_CONVERGED: return "device loop reached its iteration cap";
    case SPLIT_ERR_CUDA: return "CUDA runtime error";
    case SPLIT_ERR_OVERFLOW: return "device table capacity exceeded";
    case SPLIT_ERR_TIMEOUT: return "device-wide barrier wait timed out";
    case SPLIT_ERR_UNSUPPORTED: return "unsupported device";
    default: return "unknown status";
  }
}

namespace sg {
// first error in source order wins, as with set_status
__global__ void fold_status_kernel(WsHeader* hdr, StatusSources s, unsigned long long stamp) {
  pdl_wait();
  if (threadIdx.x != 0) return;
  hdr->stamp = stamp;
  for (int i = 0; i < s.n; ++i) {
    volatile int* q = s.p[i];
    const int v = *q;
    if (v) {
      set_status(&hdr->status, v);
      *q = 0;
    }
  }
}

int fold_status(WsHeader* hdr, const StatusSources& s, cudaStream_t st,
                unsigned long long stamp) {
  launch_pdl(fold_status_kernel, dim3(1), dim3(32), 0, st, hdr, s, stamp);
  return launch_status();
}

__global__ void clear_stages_kernel(StageHeaders s) {
  pdl_wait();
  if (threadIdx.x != 0) return;
  enter_stages(s, s.hdr->stamp);
  s.hdr->stamp = s.stamp;
}

int clear_stages(const StageHeaders& s, cudaStream_t st) {
  launch_pdl(clear_stages_kernel, dim3(1), dim3(32), 0, st, s);
  return launch_status();
}
}  // namespace sg

// The header's first words in one copy; the status word goes back to zero, which
// it nearly always is already (a clear is a launch).
static int read_header(void* workspace, void* stream, int* out_status, int* out_result) {
  cudaStream_t st = as_stream(stream);
  struct {
    int words[offsetof(WsHeader, result) / sizeof(int) + 1];
  } h;
  SG_CUDA_TRY(cudaMemcpyAsync(&h, workspace, sizeof(h), cudaMemcpyDeviceToHost, st));
  SG_CUDA_TRY(cudaStreamSynchronize(st));
  if (h.words[0] != 0) SG_CUDA_TRY(cudaMemsetAsync(workspace, 0, sizeof(int), st));
  *out_status = h.words[0];
  if (out_result) *out_result = h.words[sizeof(h) / sizeof(int) - 1];
  return SPLIT_OK;
}

extern "C" int split_workspace_status(void* workspace, void* stream, int* out_status) {
  if (!workspace || !out_status) return SPLIT_ERR_INVALID;
  return read_header(workspace, stream, out_status, nullptr);
}

extern "C" int32_t* split_workspace_result(void* workspace) {
  return workspace ? &static_cast<WsHeader*>(workspace)->result : nullptr;
}

extern "C" int split_workspace_finish(void* workspace, void* stream, int* out_status,
                                      int32_t* out_result) {
  if (!workspace || !out_status || !out_result) return SPLIT_ERR_INVALID;
  return read_header(workspace, stream, out_status, out_result);
}
