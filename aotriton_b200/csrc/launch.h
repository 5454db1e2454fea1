// Host-side declarations shared by the kernel translation units and the C-ABI layer.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>
#include <tuple>
#include <type_traits>
#include <utility>
#include "common.cuh"

namespace ab200 {

// Integer dropout threshold: keep iff (int32)philox_word > threshold.
// Restates `((dropout_p - 0.5) * 0xFFFFFFFF).to(tl.int32)` of ROCm/aotriton
// modules/flash/kernel/fwd_kernel.py:195 -- fp32 arithmetic, the literal rounds
// to 2^32 in fp32, conversion truncates toward zero and saturates.
inline int32_t dropout_threshold(float dropout_p) {
  float x = (dropout_p - 0.5f) * 4294967296.0f;
  if (!(x == x)) return 0;
  if (x >= 2147483647.0f) return 2147483647;
  if (x <= -2147483648.0f) return (int32_t)(-2147483647 - 1);
  return (int32_t)truncf(x);
}

void count_launch();

// Every CUDA runtime / driver call the launch path makes goes through this table.  Normally the
// entries forward to CUDA.  Tests can switch to a pretended sm_100 device (no GPU needed: device
// queries answer, symbol look-ups and launches are recorded and skipped) and can make the n-th call of
// any entry return an error code, to check that each failure comes back to the caller as that code
// with nothing launched after it (ab200_debug_host_calls).  No test ever makes a device fault.
enum HostCallId : int { kCallGetDevice = 0, kCallSetDevice, kCallStreamDevice, kCallDeviceAttr, kCallFuncSetSmem,
                        kCallSymbolAddress, kCallMemsetAsync, kCallLaunch, kCallEncodeTiled, kCallStreamSync,
                        kNumHostCalls };
struct HostCalls {
  cudaError_t (*get_device)(int* dev);
  cudaError_t (*set_device)(int dev);
  cudaError_t (*stream_device)(cudaStream_t st, int* dev);
  cudaError_t (*device_attr)(int* value, cudaDeviceAttr attr, int dev);
  cudaError_t (*func_set_smem)(const void* fn, int bytes);
  cudaError_t (*symbol_address)(void** ptr, const void* symbol);
  cudaError_t (*memset_async)(void* ptr, int value, size_t bytes, cudaStream_t st);
  cudaError_t (*launch)(const void* fn, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t st, bool early);
  // cuTensorMapEncodeTiled; returns a CUresult (0 = success, 100 = no encoder available)
  int (*encode_tiled)(CUtensorMap* map, CUtensorMapDataType type, cuuint32_t rank, void* base, const cuuint64_t* dims,
                      const cuuint64_t* strides, const cuuint32_t* box, const cuuint32_t* estr,
                      CUtensorMapInterleave il, CUtensorMapSwizzle sw, CUtensorMapL2promotion l2,
                      CUtensorMapFloatOOBfill fill);
  cudaError_t (*stream_sync)(cudaStream_t st);
  bool (*have_encoder)();
};
const HostCalls& host();
// true while the table pretends a device: nothing learnt from it may be remembered for real launches
bool host_pretends();

// kernel<<<grid, block, smem, st>>>(args...) through the table.  The arguments are converted to the
// kernel's exact parameter types and copied, as the launch API takes one pointer per parameter.
// `early`: set up while the grid before it still runs (h_launch).  Measured, us a pass among others, without and with: one token of 4
// sequences against 6007 keys, 32:8 heads of 128, 22.4 / 20.4; training step of 4 x 8 x 1024 x 77 of 80 86.0 / 79.6, of 16 x 12 x 391 of
// 64 with dropout 295 / 289.5; prefill of 3001 tokens 99.2 / 98.1.  Not for the general kernels, several CTAs of which share an SM:
// set up early, they fill the SMs that are free first, the longest two on the same one (fp32, 2 x 8 x 500 x 64 130.8 / 132.7).
template <bool kEarly, typename... KArgs, typename... Args>
cudaError_t launch_kernel_as(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  static_assert(sizeof...(KArgs) == sizeof...(Args), "argument count differs from the kernel's parameter list");
  std::tuple<std::remove_cv_t<std::remove_reference_t<KArgs>>...> copy(std::forward<Args>(args)...);
  void* ptrs[sizeof...(KArgs) > 0 ? sizeof...(KArgs) : 1];
  std::apply([&](auto&... a) { int i = 0; ((ptrs[i++] = (void*)&a), ...); }, copy);
  return host().launch(reinterpret_cast<const void*>(kernel), grid, block, ptrs, smem, st, kEarly);
}
template <typename... A>
cudaError_t launch_kernel(A&&... a) { return launch_kernel_as<true>(std::forward<A>(a)...); }

// which: 0 forward, 1 dK/dV, 2 dQ(+dBias), 3 both (dQ and dBias share no memory with an input).  dtype:
// ab200_dtype value.
cudaError_t launch_general(int which, int dtype, const Params& p, cudaStream_t st);
cudaError_t launch_preprocess(int dtype, const Params& p, cudaStream_t st);
cudaError_t launch_dropout_sign(int dtype, const View4& r, int batch, int heads, int rows, int cols, float dropout_p,
                                const uint64_t* seed, const uint64_t* off1, uint64_t off2, cudaStream_t st);

// tcgen05 kernels (sm100_fwd.cu / sm100_bwd.cu).  *_supported say whether the shape is
// inside the kernel's range (and tile maps can be encoded here); the launchers assume it is.  *_shape: the shape alone.
bool sm100_fwd_supported(int dtype, const Params& p);
cudaError_t launch_sm100_fwd(int dtype, const Params& p, cudaStream_t st);
// Whether the split-key kernel takes a forward that the tcgen05 family runs, and how it cuts it.
struct SplitPlan { int pieces, warps, stages, chunks; };
bool sm100_fwd_split(const Params& p, int sms, SplitPlan* plan);
bool sm100_bwd_shape(int dtype, const Params& p);
bool sm100_bwd_supported(int dtype, const Params& p);
cudaError_t launch_sm100_bwd_dkdv(int dtype, const Params& p, cudaStream_t st);
cudaError_t launch_sm100_bwd_dq(int dtype, const Params& p, cudaStream_t st);
// Fused backward: dK, dV and the dQ partials in one kernel (partials added to the fp32 accumulator
// `dq_acc`, zero on entry, contiguous in dQ's logical order), then dQ = cast(sm_scale * dq_acc).
bool sm100_bwd_fused_supported(int dtype, const Params& p);
cudaError_t launch_sm100_bwd_fused(int dtype, const Params& p, float* dq_acc, cudaStream_t st);
cudaError_t launch_postprocess(int dtype, const View4& dq, const float* acc, float scale, cudaStream_t st);
// The ticket counter of the next dK/dV launch on the current device (head dims up to 128), to be zeroed ahead of it in stream order.
cudaError_t sm100_bwd_ticket(unsigned int** ticket);
// Words the tcgen05 kernels of the current device set when a bounded wait ran out (0 = none).
// Reading synchronises the device.
unsigned int sm100_fwd_status(bool reset);
unsigned int sm100_bwd_status(bool reset);

}  // namespace ab200
