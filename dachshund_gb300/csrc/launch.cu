// Launch attributes shared by contexts on several threads.
#include <map>
#include <mutex>
#include <tuple>

#include "ds_internal.cuh"

namespace ds {

namespace {
std::mutex g_attr_mu;
std::map<std::pair<int, const void*>, size_t> g_smem;  // device, kernel -> limit set
std::map<std::tuple<int, const void*, int, size_t>, int> g_ctas;
std::mutex g_coop_mu;
std::map<int, cudaEvent_t> g_coop;  // device -> end of its last cooperative launch
}  // namespace

static void raise_smem_locked(int dev, const void* fn, size_t bytes) {
  size_t& limit = g_smem[{dev, fn}];
  if (bytes <= limit || bytes <= 48 * 1024) return;
  DS_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  limit = bytes;
}

void raise_dynamic_smem(const void* fn, size_t bytes) {
  int dev = 0;
  DS_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_attr_mu);
  raise_smem_locked(dev, fn, bytes);
}

int resident_ctas(const void* fn, int threads, size_t bytes, bool all_shared) {
  int dev = 0;
  DS_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_attr_mu);
  const auto key = std::make_tuple(dev, fn, threads, bytes);
  const auto it = g_ctas.find(key);
  if (it != g_ctas.end()) return it->second;
  int per_sm = 0, optin = 0;
  cudaFuncAttributes fa;
  DS_CUDA(cudaFuncGetAttributes(&fa, fn));
  DS_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  if (fa.sharedSizeBytes + bytes <= (size_t)optin) {
    if (all_shared)
      DS_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                   (int)cudaSharedmemCarveoutMaxShared));
    raise_smem_locked(dev, fn, bytes);
    DS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, bytes));
  }
  return g_ctas[key] = per_sm;
}

void launch_cooperative(const void* fn, int ctas, int threads, void** args, size_t bytes,
                        cudaStream_t st) {
  int dev = 0;
  DS_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_coop_mu);
  cudaEvent_t& last = g_coop[dev];
  if (last)
    DS_CUDA(cudaStreamWaitEvent(st, last, 0));
  else
    DS_CUDA(cudaEventCreateWithFlags(&last, cudaEventDisableTiming));
  DS_CUDA(cudaLaunchCooperativeKernel(fn, dim3(ctas), dim3(threads), args, bytes, st));
  DS_CHECK_LAUNCH();
  DS_CUDA(cudaEventRecord(last, st));
}

}  // namespace ds
