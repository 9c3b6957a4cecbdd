// Prints, for geometries on standard input, how the convolution planners deal them out:
//   n c k d h w f stride math   (d = 0: 2-D; padding (f - 1) / 2, dense tensors)
// Host code only; links against the library.
#include "conv_tc_shift_plan.cuh"
#include "conv_tc_wgrad_api.cuh"

#include <cstdio>
#include <cstring>

using namespace dcb;

static ConvGeom geom(int n, int c, int k, int d, int h, int w, int f, int s)
{
    ConvGeom g;
    std::memset(&g, 0, sizeof(g));
    const int in[3] = {d ? d : 1, h, w};
    g.n = n, g.c = c, g.k = k;
    for (int i = 0; i < 3; ++i)
    {
        const bool flat = i == 0 && d == 0;
        g.in[i] = in[i], g.f[i] = flat ? 1 : f, g.pad[i] = (g.f[i] - 1) / 2, g.stride[i] = flat ? 1 : s, g.dil[i] = 1;
        g.out[i] = (g.in[i] + 2 * g.pad[i] - g.f[i]) / g.stride[i] + 1;
    }
    g.xs[2] = g.ys[2] = 1;
    for (int i = 1; i >= 0; --i)
    {
        g.xs[i] = g.xs[i + 1] * g.in[i + 1];
        g.ys[i] = g.ys[i + 1] * g.out[i + 1];
    }
    g.xs_c = g.xs[0] * g.in[0], g.xs_n = g.xs_c * c;
    g.ys_c = g.ys[0] * g.out[0], g.ys_n = g.ys_c * k;
    return g;
}

int main()
{
    int v[9];
    while (std::scanf("%d %d %d %d %d %d %d %d %d", v, v + 1, v + 2, v + 3, v + 4, v + 5, v + 6, v + 7, v + 8) == 9)
    {
        const ConvGeom g = geom(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]);
        for (int tr = 0; tr < 2; ++tr)
        {
            ShTables t;
            const bool ok = ShBuilder(g, tr == 1, v[8], 148).build(&t);
            std::printf("%s %d %d %d %d\n", tr ? "bwd_data" : "fwd", ok ? 1 : 0, ok ? t.chain : 0, ok ? t.g.nsets : 0,
                        ok && simt_is_faster(g, tr == 1, t.cost / 1900.0) ? 1 : 0);
        }
        WgGeom wg;
        const bool ok = wg_geom(g, v[8], 148, &wg);
        std::printf("bwd_filter %d %d\n", ok ? 1 : 0, ok ? wg.roles : 0);
    }
    return 0;
}
