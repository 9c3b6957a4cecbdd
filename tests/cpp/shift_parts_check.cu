// Rows cut in parts that lie side by side in the lanes of the shift kernel: for layers of many
// widths, prints how many passes are laid out, in how many of them several sub-columns are parts of
// one row's width, and in how many an output is not some lane's exactly once, a position that
// an output reads is not staged, or a lane's cells leave the A slot.
// Host code only; links against the library.
#include "conv_tc_shift_plan.cuh"

#include <cstdio>
#include <cstring>

using namespace dcb;

static ConvGeom geom(int c, int k, int d, int h, int w, int f, int s)
{
    ConvGeom g;
    std::memset(&g, 0, sizeof(g));
    const int in[3] = {d ? d : 1, h, w};
    g.n = 1, g.c = c, g.k = k;
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

// Positions to the right of an output's own (or of its group's, backward with stride s) that it reads, of the tensor
// along W: forward a position is s cells, backward one cell of dy.
static int reach_of(int f, int s, bool transposed)
{
    if (!transposed)
        return (f - 1) / s;
    const int pad = (f - 1) / 2;
    int lo = f, hi = -f;
    for (int o = 0; o < s; ++o) // cells of a group
        for (int tap = 0; tap < f; ++tap)
            if ((o + pad - tap) % s == 0)
            {
                lo = std::min(lo, (o + pad - tap) / s);
                hi = std::max(hi, (o + pad - tap) / s);
            }
    return hi - lo;
}

// The kernel's walk: units, sub-columns, planes, rows, lanes.
static bool once(const ShTables& t, int f, int s, bool transposed)
{
    const ShGeom& g = t.g;
    const int reach = reach_of(f, s, transposed), row = std::min(g.tile_w, g.q_w), staged = g.ipr / g.st_w * 32;
    if (g.npack * t.per > g.pt || (g.npack - 1) * t.per + g.tile_w > TC_M)
        return false;
    // what an output reads lies in its own sub-column and is staged by an item
    for (int sub = 0; sub < g.npack; ++sub)
        for (int xx = 0; xx < row; ++xx)
            if ((sub * t.per + xx + reach) / t.per != sub || sub * t.per + xx + reach >= staged)
                return false;
    std::vector<unsigned char> seen((size_t) g.q_s * g.q_r * g.q_w, 0);
    const int sub_s = g.pack_s > 0 ? g.npack : 1, sub_r = g.pack_r > 0 ? g.npack : 1;
    for (unsigned u = 0; u < g.units / (unsigned) (g.n * g.kgroups); ++u)
    {
        const int tw = (int) (u % g.tiles_w), hb = (int) (u / g.tiles_w % g.hblks), sg = (int) (u / g.tiles_w / g.hblks);
        const int q0 = sg * g.seglen * sub_s, q1 = std::min(q0 + g.seglen, g.q_s), row0 = hb * g.th * sub_r;
        for (int q = q0; q < q1; ++q)
            for (int j = 0; j < g.th; ++j)
                for (int p = 0; p < g.npack * t.per; ++p)
                {
                    const int sub = p / t.per, xx = p % t.per, s = q + sub * g.pack_s, r = row0 + j + sub * g.pack_r, w = tw * g.tile_w + xx;
                    if (xx < g.tile_w && p < TC_M && s < g.q_s && r < g.q_r && w < g.q_w)
                        ++seen[((size_t) s * g.q_r + r) * g.q_w + w];
                }
    }
    return std::all_of(seen.begin(), seen.end(), [](unsigned char v) { return v == 1; });
}

int main()
{
    int passes = 0, parts = 0, bad = 0;
    for (int w : {16, 31, 63, 64, 65, 66, 70, 88, 96, 100, 127, 128, 129, 132, 150, 177, 192, 200, 256, 300})
        for (int flat = 0; flat < 2; ++flat)
            for (int f : {3, 5})
                for (int s = 1; s <= 2; ++s)
                    for (int tr = 0; tr < 2; ++tr)
                    {
                        ShTables t;
                        if ((!flat && f == 5) || !ShBuilder(geom(8, 24, flat ? 0 : 20, 37, w, f, s), tr == 1, DCB_MATH_FP32, 148).build(&t))
                            continue;
                        ++passes;
                        parts += t.g.npack > 1 && t.g.tiles_w > 1;
                        bad += !once(t, f, s, tr == 1);
                    }
    std::printf("%d %d %d\n", passes, parts, bad);
    return 0;
}
