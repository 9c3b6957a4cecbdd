// Backward filter with stride 2 along W.
#include "conv_tc_wgrad.cuh"

namespace dcb
{

int32_t wg_launch_s2(const WgGeom& g, int al, int rkw, const float* x, const float* dy, float* part, int* status,
                     cudaStream_t stream)
{
    switch (g.kwg)
    {
    case 1: return wg_launch_at<2, 1>(g, al, rkw, x, dy, part, status, stream);
    case 3: return wg_launch_at<2, 3>(g, al, rkw, x, dy, part, status, stream);
    default: return wg_launch_at<2, 5>(g, al, rkw, x, dy, part, status, stream);
    }
}

} // namespace dcb
