// deb_internal.h -- library-internal declarations shared by the CUDA
// translation units (not part of the C ABI).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <mutex>

#include "deb_core.cuh"

struct deb_plan {
  deb::Dims D;
  int dense, return_full, nout, exec_mode;
  int max_modes, nsm;
  long slot_len, dense_len;
  // lane mode
  int lane_blocks, lane_slots;
  // warp mode
  int block_warps, warp_blocks, warp_smem, warp_k_global, warp_per_sm;
  // grouped plans (deb_plan_create_grouped): modes per group, groups in flight
  // with the slots in shared memory (0: they don't fit) and in global memory
  int group_size, group_shared, group_global;
  long warp_smem_bytes;
  double* kws;      // warp mode: stage vectors in global memory
  double* ws;       // lane slots (or warp slots when shared memory is too small)
  double* dws;      // dense matrices
  int* queue;
  int* order_dev;   // replay order (max_modes ints)
  const int* user_order;   // deb_plan_set_order
  int user_order_n;
  size_t ws_bytes;
  // adjoint plans (deb_plan_create_adjoint): blocks in flight, states per
  // segment, per-block workspace (doubles) and its array
  int adj, adj_blocks, adj_seg_cap;
  long adj_wslot;
  // launch shape with one block per SM, with two: dynamic shared memory (bytes) and
  // what of an item's state lives there (deb_adjoint.cu)
  long adj_smem[2];
  int adj_level[2];
  double* adj_ws;
};


namespace deb_internal {

using PFN_ctxGetCurrent = CUresult (*)(CUcontext*);
using PFN_ctxGetId = CUresult (*)(CUcontext, unsigned long long*);

// Unique id of the current thread's CUDA context (never reused within a
// process), 0 if it cannot be determined.  The driver entry points are found
// through the runtime, so the library needs no link to libcuda.
inline unsigned long long current_ctx_id() {
  static PFN_ctxGetCurrent get_cur = nullptr;
  static PFN_ctxGetId get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_cur = (PFN_ctxGetCurrent)f;
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = (PFN_ctxGetId)f;
  });
  if (!get_cur || !get_id) return 0;
  CUcontext ctx = nullptr;
  if (get_cur(&ctx) != CUDA_SUCCESS || !ctx) return 0;
  unsigned long long id = 0;
  if (get_id(ctx, &id) != CUDA_SUCCESS) return 0;
  return id + 1;   // 0 stays "unknown"
}

// The dynamic shared-memory limit of one kernel on each device.  The attribute
// belongs to the kernel, so it is raised under a lock and never lowered: a
// launch on another thread, or a plan made earlier, may need the larger value.
// After a device reset (or with another context current) it is set again.
struct SmemLimit {
  std::mutex mu;
  unsigned long long ctx[64] = {0};
  long bytes[64] = {0};
  template <class Kernel>
  cudaError_t raise(Kernel* kernel, long want) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long id = current_ctx_id();
    std::lock_guard<std::mutex> lock(mu);
    const bool kept = dev >= 0 && dev < 64, same = kept && ctx[dev] == id;
    if (same && id != 0 && bytes[dev] >= want) return cudaSuccess;
    if (want < 48 * 1024) want = 48 * 1024;   // the limit that needs no attribute
    if (same && want < bytes[dev]) want = bytes[dev];
    const cudaError_t rc = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)want);
    if (rc == cudaSuccess && kept) { ctx[dev] = id; bytes[dev] = want; }
    return rc;
  }
};

}  // namespace deb_internal
