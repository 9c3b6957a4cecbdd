// Backward filter with stride 1 along W.
#include "conv_tc_wgrad.cuh"

namespace dcb
{

int32_t wg_launch_s1(const WgGeom& g, int al, int rkw, const float* x, const float* dy, float* part, int* status,
                     cudaStream_t stream)
{
    switch (g.kwg)
    {
    case 1: return wg_launch_at<1, 1>(g, al, rkw, x, dy, part, status, stream);
    case 3: return wg_launch_at<1, 3>(g, al, rkw, x, dy, part, status, stream);
    default: return wg_launch_at<1, 5>(g, al, rkw, x, dy, part, status, stream);
    }
}

} // namespace dcb
