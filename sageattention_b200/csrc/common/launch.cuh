// Kernel launches with programmatic stream serialisation, and the shared-memory opt-in done once.
//
// Every kernel of the library is launched so that its CTAs may start while the kernel before it on the
// stream drains: barrier initialisation, tensor-memory allocation and descriptor fetches then overlap
// the predecessor's tail instead of following it.  The rules that make this safe:
//   * every thread executes griddep_wait() before its first access to global memory (L2 prefetch hints
//     excepted: L2 is the point of coherence); it returns when all earlier work of the stream is
//     complete and visible, and since no kernel finishes without it, completion is transitive;
//   * a kernel that allocates tensor memory calls griddep_launch() only after its allocation, so a
//     dependent that starts on the same SM cannot take columns its predecessor still waits for.
// One exception, the late wait: a kernel that needs nothing of the kernel P launched directly before it may
// take the operands that were there before P at once and call griddep_wait() at its END, where it keeps
// completion transitive.  It then starts as soon as P has signalled, and rests on three conditions:
//   * P executes griddep_wait() BEFORE griddep_launch(): its signal says that everything before P is
//     complete.  (P may be a late waiter itself, directly behind such a kernel: it starts after that signal.)
//     Swapping the two lines in P would be a race that no test is sure to show;
//   * one host call launches both.  A launch that another thread puts between them does no harm, it cannot start
//     before P's signal either; but only a caller that launches P knows that nothing it needs comes after P;
//   * it reads nothing that P writes and writes nothing that P reads or writes.
// What such a kernel reads early was complete, and in L2, before its grid began; no wait of its own stands between.
// Checked on a B200: grids that start early on SMs whose L1 had held the words, after a grid on another SM rewrote
// them, read none of 9.7e9 stale.  A fence.acq_rel.gpu at the start instead costs every CTA ~0.3 us: backward of
// a packed row of 16384 tokens H32 D128 1357 -> 1375 us.
// Late waiters, and what each stands behind:
//   bwd_dq_kernel   behind bwd_dkdv_kernel (nvfp4_bwd_hp)
//   bwd4_kernel     passes after the first, behind bwd4_kernel (nvfp4_bwd_fp4)
//   decode_kernel   behind window_mma_kernel or window_attention_kernel (nvfp4_decode_window)
#pragma once
#include <cuda_runtime.h>
#include <atomic>
#include <stdint.h>
#include "abi.cuh"

namespace nvfp4 {

__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Start of a kernel that can be a late waiter; its end calls griddep_wait() if `late`.
__device__ __forceinline__ void griddep_start(bool late) {
  if (!late) griddep_wait();
}

// What is done once per kernel and device: a fixed open-addressing table of kernel addresses (the library has fewer
// kernels than slots), lock-free, so that a launch pays a look-up (~20 ns) instead of the driver call.  Two threads may
// both be first; what they do is the same.
struct KernelTable {
  static constexpr int kSlots = 512;
  std::atomic<const void*> keys[kSlots];
  std::atomic<uint64_t> devices[kSlots];
  // the slot's devices, or null where the table is full
  std::atomic<uint64_t>* find(const void* kern) {
    uint32_t i = (uint32_t)((reinterpret_cast<uintptr_t>(kern) >> 4) * 2654435761u) % kSlots;
    for (int probe = 0; probe < kSlots; ++probe, i = (i + 1) % kSlots) {
      const void* k = keys[i].load(std::memory_order_acquire);
      if (k == nullptr && keys[i].compare_exchange_strong(k, kern, std::memory_order_acq_rel)) k = kern;
      if (k == kern) return &devices[i];
    }
    return nullptr;
  }
};

// cudaFuncSetAttribute(attr, value) of a kernel; `value` must be the same in every call for a kernel and attribute.
template <cudaFuncAttribute kAttr>
cudaError_t kernel_attribute(const void* kern, int value) {
  static KernelTable table;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  std::atomic<uint64_t>* seen = table.find(kern);
  if (seen != nullptr && (seen->load(std::memory_order_acquire) & bit)) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, kAttr, value);
  if (e == cudaSuccess && seen != nullptr) seen->fetch_or(bit, std::memory_order_acq_rel);
  return e;
}

inline int allow_smem(const char* what, const void* kern, int bytes) {
  const cudaError_t e = kernel_attribute<cudaFuncAttributeMaxDynamicSharedMemorySize>(kern, bytes);
  if (e != cudaSuccess) return fail((int)e, "%s: smem attribute: %s", what, cudaGetErrorString(e));
  return 0;
}

// For kernels that stream through L1: at most `kStreamSmem` percent of it as shared memory (three blocks of the V^T
// packers).  A load in flight holds a line of L1, and an SM keeps the split that the kernel before it asked for: behind the
// forward, whose 202 KB leave 28 of L1, the packs of a prompt Z4 S8192 took 119 us instead of 92 (prompt S12289 D256 in all
// 675 -> 663).  A hint, not checked.
constexpr int kStreamSmem = 45;
inline void prefer_l1(const void* kern) {
  if (kernel_attribute<cudaFuncAttributePreferredSharedMemoryCarveout>(kern, kStreamSmem) != cudaSuccess) cudaGetLastError();
}

// Clusters of `size` CTAs (1 to 8, else 0) of a kernel that are resident at once.  Of kernels whose shared memory leaves room
// for one CTA per SM the answer depends on the size alone and is asked once per device; of others on every call.
// allow_smem() has been called for `kern`.
constexpr int kSmemPerSm = 228 * 1024;
inline int cluster_slots(const void* kern, unsigned threads, int smem, int sms, int size) {
  static std::atomic<int> known[64][9];
  if (size < 1 || size > 8) return 0;
  int dev = 0;
  const bool keep = 2 * smem > kSmemPerSm && cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64;
  int n = keep ? known[dev][size].load(std::memory_order_relaxed) : 0;
  if (n > 0) return n;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = size;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1, 1, size);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
    cudaGetLastError();
    return sms / size;
  }
  if (keep) known[dev][size].store(n, std::memory_order_relaxed);
  return n;
}
// the same for 1, 2, 4 and 8
inline void cluster_slots(const void* kern, unsigned threads, int smem, int sms, int (&slots)[4]) {
  for (int i = 0; i < 4; ++i) slots[i] = cluster_slots(kern, threads, smem, sms, 1 << i);
}

// Launch with programmatic stream serialisation; launch_cluster: clusters of `cluster` CTAs along z.
template <typename... P, typename... A>
int launch_cluster(const char* what, void (*kern)(P...), dim3 grid, unsigned cluster, unsigned threads, size_t smem,
                   cudaStream_t st, A&&... args) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cluster > 1) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = cluster;
    cfg.numAttrs = 2;
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, P(args)...);
  if (e != cudaSuccess) {
    cudaGetLastError();          // the failure is reported here; leave no sticky code behind
    return fail((int)e, "%s: %s", what, cudaGetErrorString(e));
  }
  return 0;
}

template <typename... P, typename... A>
int launch(const char* what, void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A&&... args) {
  return launch_cluster(what, kern, grid, 1, threads, smem, st, static_cast<A&&>(args)...);
}

// launch() of a kernel that streams through L1, if its blocks' shared memory leaves three of them room within the hint
template <bool kFits = true, typename... P, typename... A>
int launch_streaming(const char* what, void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A&&... args) {
  if constexpr (kFits) prefer_l1(reinterpret_cast<const void*>(kern));
  return launch_cluster(what, kern, grid, 1, threads, smem, st, static_cast<A&&>(args)...);
}

}  // namespace nvfp4
