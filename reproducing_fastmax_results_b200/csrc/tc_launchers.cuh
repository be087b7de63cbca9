// Entry points of the tcgen05 / TMA kernels.  Each returns FASTMAX_TC_NOT_HANDLED when the problem is
// outside what the tensor-core kernels cover, and the caller then runs the CUDA-core engine.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>

#include <memory>

#include "../../include/fastmax_b200.h"

namespace fm {
enum { FASTMAX_TC_NOT_HANDLED = -1 };
size_t tc_forward_workspace(const fastmax_problem* pb, const fastmax_forward_args* a);
size_t tc_backward_workspace(const fastmax_problem* pb, const fastmax_backward_args* a);
// Whether the tensor-memory kernels take the call (they may still hand it back at run time when the copy engine
// cannot describe a tensor's layout; the CUDA-core engine then runs it).
bool tc_takes_forward(const fastmax_problem* pb, const fastmax_forward_args* a);
bool tc_takes_backward(const fastmax_problem* pb, const fastmax_backward_args* a);
// Bytes of the per-segment moment arrays a segmented tensor-memory call reads or writes (0: the call is not segmented).
size_t tc_key_moments_bytes(const fastmax_problem* pb, const fastmax_forward_args* a);
size_t tc_grad_moments_bytes(const fastmax_problem* pb, const fastmax_backward_args* a);
int tc_forward(const fastmax_problem* pb, const fastmax_forward_args* a, void* ws, size_t ws_bytes, cudaStream_t st);
int tc_backward(const fastmax_problem* pb, const fastmax_backward_args* a, void* ws, size_t ws_bytes, cudaStream_t st);
// Reads (and clears) the device-side error word the bounded waits of the tensor-core kernels set.
int tc_device_status(int* out);
// Copies (and clears) the per-wait-site give-up counters (index = error code & 255).
int tc_wait_histogram(int* out, int n);
// Launches the test-only kernel that lets a bounded wait of `cycles` SM clocks run out and records wait site `code`.
int tc_wait_selftest(long long cycles, int code, cudaStream_t st);

// bf16 (batch, head, token, cols) view -> 4-D tensor map with a [box_rows x box_cols] box (columns past `cols` read as
// zero); f32: the elements are float32; false when the copy engine cannot describe the view
bool tc_make_map(CUtensorMap* m, const fastmax_tensor& t, int batch, int heads, int n, int box_cols, int box_rows, bool swizzle128,
                 int cols, bool f32 = false);

size_t tc_moments_scratch(const fastmax_problem* pb, int n);
cudaError_t tc_moments(const fastmax_problem* pb, const fastmax_tensor& x, const fastmax_tensor& y, int n, bool dop, int seg_tokens,
                       const float* init, float* state, void* xt, cudaStream_t st);

// A second stream for work that is independent of what the caller's stream gets meanwhile: forked from it here, joined back
// by join() (or the destructor).  The caller's own stream when side streams are off.  Calls made on `side` must carry
// FASTMAX_FLAG_SINGLE_STREAM: the device's side streams are leased until the join.
struct SideBranch {
  SideBranch(const fastmax_problem* pb, cudaStream_t st);
  ~SideBranch();
  cudaError_t join();
  cudaStream_t main, side;

 private:
  struct Lease;
  std::shared_ptr<Lease> lease;
};

// shared with the C-ABI translation unit
int report_cuda_error(cudaError_t e);  // remembers e for fastmax_last_cuda_error(), returns FASTMAX_ERR_CUDA
// acc: [batch*heads][n][acc_ld] float32 (acc_ld <= 0: dense, acc_ld = d)
int launch_cast_out(const fastmax_problem* pb, const float* acc, int n, const fastmax_tensor* out, cudaStream_t st, int acc_ld = 0);
int launch_finalize_fwd(const fastmax_problem* pb, const fastmax_forward_args* a, const float* oacc, cudaStream_t st);
}  // namespace fm
