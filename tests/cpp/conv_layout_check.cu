// How layers on standard input are laid out:
//   n c k d h w fd fh fw pd ph pw s math   (d = 0: 2-D; dense tensors, 148 SMs)
// prints "sweep ok slots" (A slots of a converter group of the sweep kernel) and per pass of the shift
// kernel "fwd ok npack tiles_w stage" / "bwd_data ..." (sub-columns side by side, tiles of a row, bytes
// that a warp stages for bulk stores).  Host code only; links against the library.
#include "conv_tc.cu"
#include "conv_tc_shift_plan.cuh"

#include <cstdio>

using namespace dcb;

int main()
{
    int n, c, k, in[3], f[3], pad[3], s, math;
    while (std::scanf("%d %d %d %d %d %d %d %d %d %d %d %d %d %d", &n, &c, &k, in, in + 1, in + 2, f, f + 1, f + 2, pad, pad + 1,
                      pad + 2, &s, &math)
           == 14)
    {
        ConvGeom g;
        std::memset(&g, 0, sizeof(g));
        g.n = n, g.c = c, g.k = k;
        for (int i = 0; i < 3; ++i)
        {
            const bool flat = i == 0 && in[0] == 0;
            g.in[i] = flat ? 1 : in[i], g.f[i] = flat ? 1 : f[i], g.pad[i] = flat ? 0 : pad[i], g.stride[i] = flat ? 1 : s;
            g.dil[i] = 1;
            g.out[i] = (g.in[i] + 2 * g.pad[i] - g.f[i]) / g.stride[i] + 1;
        }
        g.xs[2] = g.ys[2] = 1;
        for (int i = 1; i >= 0; --i)
            g.xs[i] = g.xs[i + 1] * g.in[i + 1], g.ys[i] = g.ys[i + 1] * g.out[i + 1];
        g.xs_c = g.xs[0] * g.in[0], g.xs_n = g.xs_c * c;
        g.ys_c = g.ys[0] * g.out[0], g.ys_n = g.ys_c * k;
        SwGeom sw;
        const bool sweep = sw_geom(g, math, &sw);
        std::printf("sweep %d %d\n", sweep ? 1 : 0, sweep ? sw.a_slots / sw.groups : 0);
        for (int tr = 0; tr < 2; ++tr)
        {
            ShTables t;
            const bool ok = ShBuilder(g, tr == 1, math, 148).build(&t);
            std::printf("%s %d %d %d %d\n", tr ? "bwd_data" : "fwd", ok ? 1 : 0, ok ? t.g.npack : 0, ok ? t.g.tiles_w : 0,
                        ok ? t.g.stage : 0);
        }
    }
    return 0;
}
