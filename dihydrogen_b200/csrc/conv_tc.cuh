// Interface of the tcgen05 sweep kernel (forward, few input channels) and of the
// tcgen05 backward filter.
#pragma once

#include "conv_simt.cuh"

namespace dcb
{

struct TcPlan;

// Tensor-core state for the forward geometry `fwd` and its backward filter; *out
// stays null (and DCB_OK is returned) when neither kernel covers the geometry.
int32_t tc_plan_create(const ConvGeom& fwd, int math_mode, TcPlan** out);
void tc_plan_destroy(TcPlan* p);
bool tc_has_sweep(const TcPlan* p);
bool tc_has_bwd_filter(const TcPlan* p);
// `status`: device word that a kernel sets when a bounded wait expires.
// y = alpha * conv(x, w), optionally with the per-filter sums and sums of squares
// of y.  DCB_UNSUPPORTED, with nothing launched, when the kernel does not cover
// the plan or x's alignment.
int32_t tc_sweep_fwd(TcPlan* p, float alpha, const float* x, const float* w,
                     float* y, int* status, cudaStream_t stream,
                     float* sums = nullptr, float* sqsums = nullptr);
int32_t tc_conv_bwd_filter(TcPlan* p, float alpha, const float* x,
                           const float* dy, float beta, float* dw,
                           int* status, cudaStream_t stream);

} // namespace dcb
