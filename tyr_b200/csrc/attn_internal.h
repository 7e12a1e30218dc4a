// Internal launch interface shared by the .cu files of the attention library.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/tyr_b200_attn.h"

namespace tyr {

// Launch with programmatic stream serialisation: the kernel's CTAs may become resident while the
// grid before it in the stream is still draining.  Every kernel launched this way executes
// griddepcontrol.wait (grid_dependency_wait) in every thread block before it touches memory that an
// earlier grid may write or still read, so only its launch latency and set-up overlap (and reads such memory by ordinary
// loads: the read-only path is for what no one writes during a kernel's lifetime, which begins earlier here).  A grid lets
// its successor start by griddepcontrol.launch_dependents (grid_launch_dependents).  The one exception
// is the dQ kernel of the backward, which runs next to the dK/dV kernel, reads its inputs from L2 and waits at its end.
template <class... P, class... A>
inline cudaError_t launch_kernel(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, unsigned cluster_x,
                                 bool overlap, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (overlap) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster_x > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = cluster_x;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <class... P, class... A>
inline cudaError_t launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, unsigned cluster_x,
                                     A&&... args) {
  return launch_kernel(kernel, grid, block, smem, st, cluster_x, true, static_cast<A&&>(args)...);
}

// From this many query rows or keys on, the order of the sums behind a (batch, head)'s results is the same in
// every causal launch, whatever else is in the batch: its bits are those of a call of its own, as the header promises.
// Below it a launch with too few work items for the SMs may cut a row's keys, or a key's query rows, over more of
// the device.  The line is that promise, not where the gain ends.  One prompt, forward, cut / uncut: 2048 rows, 6 heads of
// 64 17.5 / 29.2 us, 16/8 heads of 128 24.7 / 33.7, 3072 rows 24.1 / 41.3 and 46.8 / 46.8; 2047 rows are cut: 17.5 and 24.7.
constexpr int kOneOrderSeq = 2048;

// Per-device state owned by api.cu.
struct DeviceState {
  int* status = nullptr;  // device word the kernels' bounded waits OR into
  bool ready = false;
};
DeviceState* device_state(int device);  // lazily created; nullptr on failure
void count_launch(int n = 1);
int sm_count();  // SMs of the current device (148 when it cannot be asked)
// Cycles a single in-kernel barrier wait may take before its CTA gives up (api.cu; the default
// unless a test shortened it).
long long wait_limit_cycles();
// ptx_sm100.cuh users only: a one-warp kernel whose only barrier is never arrived at, so that its
// bounded wait runs out after `limit_cycles` (stalled_wait.cu).
int launch_stalled_wait(long long limit_cycles, int* status, cudaStream_t st);

// prefill_sm100.cu — tcgen05/TMA kernel, bf16, head_dim in {64,128}.
int launch_prefill_sm100(const TyrAttnPrefillArgs& a, float scale, int* status, cudaStream_t st);
long long prefill_split_workspace_bytes(const TyrAttnPrefillArgs& a);  // 0: the launch would not split
// 128-byte-swizzled 64 x 128 box map over a bf16 [batch, heads, seq, d] tensor with element strides
// {batch, head, seq}; encoded maps are cached per thread (prefill_sm100.cu).
int make_tile_map(CUtensorMap* m, const void* ptr, int batch, int heads, int seq, int d, const int64_t* stride);
// backward_sm100.cu — tcgen05/TMA kernels, bf16, head_dim in {64,128}.
size_t backward_workspace_bytes(int batch, int n_head, int q_seq);
int launch_backward_sm100(const TyrAttnBackwardArgs& a, float scale, int* status, cudaStream_t st);
// check_fp32.cu — fp32-FMA kernel, bf16 or fp32 I/O, any head_dim <= 256.
int launch_prefill_check(const TyrAttnPrefillArgs& a, float scale, cudaStream_t st);
// decode_splitkv.cu
size_t decode_workspace_bytes(int batch, int n_head, int head_dim, int max_kv_seq, int max_splits);
int decode_num_splits(int max_kv_seq, int max_splits, int* chunk_len);
int launch_decode(const TyrAttnDecodeArgs& a, float scale, cudaStream_t st);
// Unmasked forward calls with few query rows per KV head (group * q_seq), served by the decode kernel.
bool few_rows_call(const TyrAttnPrefillArgs& a);
size_t few_rows_workspace_bytes(const TyrAttnPrefillArgs& a);  // 0: the launch would not use one
int launch_few_rows(const TyrAttnPrefillArgs& a, float scale, int* status, cudaStream_t st);
int launch_merge2(const float* o_a, const float* lse_a, const float* o_b, const float* lse_b,
                  float* o_out, float* lse_out, int64_t rows, int head_dim, cudaStream_t st);

// qk_prologue.cu
int launch_qk_prologue(const TyrAttnPrologueArgs& a, int* status, cudaStream_t st);

}  // namespace tyr
