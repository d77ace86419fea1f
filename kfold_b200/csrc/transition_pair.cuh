// Transition of bf16 rows of 128 or 256 channels in one kernel (declarations).
#pragma once
#include "common.cuh"

namespace kfb {

// Whether launch_transition_pair takes these operands (kfb_transition_fwd's): contiguous rows, 16-byte aligned, a hidden width of whole
// blocks of 128, a device that holds CTA pairs.
bool transition_pair_ok(const void* x, const void* w_swiglu, const void* w_out, const void* out, const void* resid, long long rows, int c,
                        int hidden, int dtype);
// Whether it then takes less of the GPU's time than the three launches.
bool transition_pair_is_faster(long long rows, int c, int hidden);
// out may be x, and so may resid.  w_static: the weights were written before the launch before this one.
int launch_transition_pair(cudaStream_t stream, const void* x, const float* ln_w, const float* ln_b, const void* w_swiglu, const void* w_out,
                           void* out, const void* resid, long long rows, int c, int hidden, float eps, int w_static);

}  // namespace kfb
