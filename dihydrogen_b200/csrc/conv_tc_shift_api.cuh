// Interface of the shift kernel (conv_tc_shift.cuh).
#pragma once

#include "conv_simt.cuh"

namespace dcb
{

struct ShPlan;

// Tables and device buffers for one direction of a convolution (transposed:
// backward data).  False, with *status DCB_OK, when the kernel does not cover
// the geometry.
bool sh_plan_create(const ConvGeom& g, bool transposed, int math_mode, ShPlan** out, int32_t* status);
void sh_plan_destroy(ShPlan* p);
// the epilogue can return per-filter sums and sums of squares of the output
bool sh_has_stats(const ShPlan* p);
// the planner's estimate of a launch, in microseconds (within a fifth or so)
double sh_estimate(const ShPlan* p);
// operands as three bf16 parts, six products
bool sh_bf16_split(const ShPlan* p);
// y = alpha * conv(x, w) + beta * y (transposed: x is dy, y is dx).  `status` is
// set by the kernel when a bounded wait expires.  sums / sqsums: only where
// sh_has_stats, with beta = 0.
int32_t sh_conv(ShPlan* p, float alpha, const float* x, const float* w, float beta, float* y, int* status,
                cudaStream_t stream, float* sums = nullptr, float* sqsums = nullptr);

} // namespace dcb
