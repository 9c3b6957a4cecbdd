// Tensor memory of the shift kernel: for layers of every pair of stride and filter, prints how many
// passes the planner lays out, in how many of them the epilogue fetches columns beyond the
// accumulators, and in how many it fetches one that the set-up does not zero (or that is not there).
// Host code only; links against the library.
#include "conv_tc_shift_plan.cuh"

#include <cstdio>
#include <cstring>

using namespace dcb;

static ConvGeom geom(int c, int k, const int (&in)[3], const int (&f)[3], const int (&s)[3])
{
    ConvGeom g;
    std::memset(&g, 0, sizeof(g));
    g.n = 2, g.c = c, g.k = k;
    for (int i = 0; i < 3; ++i)
    {
        g.in[i] = in[i], g.f[i] = f[i], g.pad[i] = (f[i] - 1) / 2, g.stride[i] = s[i], g.dil[i] = 1;
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

// One past the last column that the epilogue's walk over blocks, cells and filters fetches.
static int fetched(const ShGeom& g)
{
    int end = 0;
    auto fetch = [&](int column) { end = std::max(end, column + (g.nsets - 1) * g.set_off + 16); };
    for (int j = 0; j < g.th; ++j)
        for (int slot = 0; slot < g.ns; ++slot)
        {
            const int block = j * g.rowst + slot * g.blk;
            for (int ew = 0; ew < g.e_w; ++ew)
                if (g.nb < 16)
                    for (int c0 = 0; c0 < g.e_s * g.e_r * g.nb; c0 += 16)
                        fetch(block + ew * g.woff + c0);
                else
                    for (int cell = 0; cell < g.e_s * g.e_r; ++cell)
                        for (int k0 = 0; k0 < g.nb; k0 += 16)
                            fetch(block + ew * g.woff + cell * g.nb + k0);
        }
    return end;
}

int main()
{
    int passes = 0, beyond = 0, bad = 0;
    for (int d : {1, 12})
        for (int f = 1; f <= 5; ++f)
            for (int strides = 0; strides < 8; ++strides)
                for (int c : {1, 4, 5, 8, 12, 20})
                    for (int math : {DCB_MATH_FP32, DCB_MATH_TF32, DCB_MATH_BF16})
                        for (int tr = 0; tr < 2; ++tr)
                        {
                            const int flat = d == 1;
                            if (flat && (strides & 1))
                                continue;
                            const int in[3] = {d, 20, 70}, fs[3] = {flat ? 1 : f, f, f},
                                      st[3] = {1 + (strides & 1), 1 + (strides >> 1 & 1), 1 + (strides >> 2)};
                            ShTables t;
                            if (!ShBuilder(geom(tr ? c : 16, tr ? 16 : c, in, fs, st), tr == 1, math, 148).build(&t))
                                continue;
                            // (the kernel zeroes in steps of 16, from column 0)
                            const int zeroed = (sh_columns(t.g) + 15) / 16 * 16, end = fetched(t.g);
                            ++passes;
                            beyond += end > t.g.set_off * t.g.nsets;
                            bad += end > zeroed || zeroed > (int) TC_TMEM_COLS;
                        }
    std::printf("%d %d %d\n", passes, beyond, bad);
    return 0;
}
