// Entry points of the pairwise tcgen05 kernels (pair_kernels.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include "../../include/fastmax_b200.h"

namespace fm {
// Whether the pairwise kernels take the call: allowed by the caller, the cheaper form, and in a layout the copy engine reads.
bool pair_takes_forward(const fastmax_problem* pb, const fastmax_forward_args* a);
bool pair_takes_backward(const fastmax_problem* pb, const fastmax_backward_args* a);
// Moment arrays that a call on long sequences hands from forward to backward: packed window states, a form of their own.  Whether
// the forward call of these arguments writes them when it is asked for key moments, a requested final state aside; their
// bytes, which are those of no array of segment sums; and whether a backward call reads them.
bool pair_packs_key_moments(const fastmax_problem* pb, const fastmax_forward_args* a);
size_t pair_key_moments_bytes(const fastmax_problem* pb);
bool pair_reads_key_moments(const fastmax_problem* pb, const fastmax_backward_args* a);
size_t pair_forward_workspace(const fastmax_problem* pb, const fastmax_forward_args* a);
size_t pair_backward_workspace(const fastmax_problem* pb, const fastmax_backward_args* a);
int pair_forward(const fastmax_problem* pb, const fastmax_forward_args* a, void* ws, cudaStream_t st);
int pair_backward(const fastmax_problem* pb, const fastmax_backward_args* a, void* ws, cudaStream_t st);
// Device-side error word and per-wait-site give-up counters (see tc_device_status / tc_wait_histogram, which include them).
int pair_status(int* out);
int pair_wait_histogram(int* out, int n);
}  // namespace fm
