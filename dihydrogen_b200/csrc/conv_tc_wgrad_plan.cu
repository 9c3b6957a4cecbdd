// Backward filter: how a convolution is dealt out.  Host code only: needs no device.
#include "conv_tc_wgrad_api.cuh"

#include "dcb.h"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace dcb
{

namespace
{

// clocks of one instruction of width n (measured, shared-memory operands)
double wg_mma_cost(int n)
{
    const double a = n / 2.0, b = 32.0 + n / 4.0;
    return a > b ? (a > 45.5 ? a : 45.5) : (b > 45.5 ? b : 45.5);
}

// Updates of an accumulator between flushes.  A chain of truncating updates is off by 1.5e-8 to
// 2e-8 each (1.8e-6 to 2.5e-6 with WG_CHAIN), fp32 FMAs over n positions, as the CUDA-core kernel deals them
// out, by 1.4e-9 sqrt(n) and more where there are many sums.  Strided layers and rows that
// cannot be read in aligned 16-byte pieces are held to that: 16 -> 16, 24 x 40 x 67, 1.8e-6
// with WG_CHAIN, 6.4e-7 like this, 7.4e-7 with FMAs.  The others are only where they are small: with 64 updates
// (1.2e-6) 4 -> 16 would take 1125 us instead of 1053 on 256^3, 162 instead of 149 on 128^3.
int wg_chain(const ConvGeom& cg)
{
    const bool aligned = ((cg.xs[0] | cg.xs[1] | cg.xs_c | cg.xs_n | cg.ys[0] | cg.ys[1] | cg.ys_c | cg.ys_n) & 3) == 0;
    const bool strided = cg.stride[0] > 1 || cg.stride[1] > 1 || cg.stride[2] > 1;
    const double n = 0.1 * std::sqrt((double) cg.n * cg.out[0] * cg.out[1] * cg.out[2]),
                 sums = aligned ? 1.0 : std::sqrt(std::max(1.0, cg.k * (double) cg.c / 64)),
                 least = aligned && !strided ? 64.0 : 16.0;
    return (int) std::min((double) WG_CHAIN, std::max(least, n * sums));
}

// One way to deal out the work; false when it does not fit.
bool wg_layout(const ConvGeom& cg, WgGeom* out, int cgp, int kwg, int kdg, int kg, int B, int PW, bool ring, int sms, double* cost)
{
    WgGeom& g = *out;
    const int sh = cg.stride[1], fh = cg.f[1];
    auto groups = [](int total, int per) { return (total + per - 1) / per; };
    g.cg = cgp, g.kwg = kwg, g.kdg = kdg, g.kg = kg;
    g.ncg = groups(cg.c, cgp), g.nkw = groups(cg.f[2], kwg), g.nkd = groups(cg.f[0], kdg), g.nkg = groups(cg.k, kg);
    g.roles = g.ncg * g.nkd * g.nkg;
    g.kgp = (kg + 7) / 8 * 8;
    g.n8 = 2 * g.kgp;
    g.r8 = (2 * cgp * kwg + 7) / 8 * 8;
    if (g.r8 > 128 || g.n8 > 256 || g.roles > 4096)
        return false;
    g.B = B;
    g.X = (B - 1) * sh + fh;
    if (g.X > 255)
        return false;
    g.A = 128 / g.r8 < g.X ? 128 / g.r8 : g.X;
    g.PW = PW;
    g.Q = PW / 4;
    // tiles and accumulator blocks of one kd plane
    auto b_range = [&](int a0, int* lo, int* hi) {
        const int num = a0 - (fh - 1);
        *lo = num <= 0 ? 0 : (num + sh - 1) / sh;
        *hi = (a0 + g.A - 1) / sh < B - 1 ? (a0 + g.A - 1) / sh : B - 1;
    };
    int dlo[2] = {1 << 20, 1 << 20}, dhi[2] = {-(1 << 20), -(1 << 20)};
    for (int a0 = 0; a0 < g.X; a0 += g.A)
    {
        int lo, hi;
        b_range(a0, &lo, &hi);
        const int r = a0 % sh;
        if (hi < lo)
            continue;
        dlo[r] = lo - a0 / sh < dlo[r] ? lo - a0 / sh : dlo[r];
        dhi[r] = hi - a0 / sh > dhi[r] ? hi - a0 / sh : dhi[r];
    }
    g.nblocks = 0;
    g.nclasses = sh;
    for (int r = 0; r < sh; ++r)
    {
        g.class_lo[r] = dlo[r];
        g.class_n[r] = dhi[r] >= dlo[r] ? dhi[r] - dlo[r] + 1 : 0;
        g.class_col[r] = g.nblocks * g.n8;
        g.nblocks += g.class_n[r];
    }
    g.kd_cols = g.nblocks * g.n8;
    g.sum_col = kdg * g.kd_cols;
    if (g.sum_col + kdg * g.nblocks * g.kgp > (int) TC_TMEM_COLS)
        return false;
    g.ntiles = 0;
    int hits[512] = {0}, max_hits = 1; // updates of a block per k-step
    double mma = 0;
    for (int a0 = 0; a0 < g.X; a0 += g.A)
    {
        int lo, hi;
        b_range(a0, &lo, &hi);
        const int r = a0 % sh, most = 256 / g.n8;
        for (int b = lo; b <= hi; b += most)
        {
            const int nb = hi - b + 1 < most ? hi - b + 1 : most;
            if (g.ntiles == WG_MAX_TILES)
                return false;
            WgTile& t = g.tiles[g.ntiles++];
            t.a16 = (uint32_t) (a0 * g.r8);
            t.b16 = (uint32_t) (b * g.n8);
            t.dcol = (uint32_t) (g.class_col[r] + (b - a0 / sh - g.class_lo[r]) * g.n8);
            t.idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((128u >> 4) << 24) | ((uint32_t) (nb * g.n8 >> 3) << 17);
            mma += wg_mma_cost(nb * g.n8);
            for (int i = 0; i < nb; ++i)
            {
                int& h = hits[t.dcol / g.n8 + i];
                max_hits = ++h > max_hits ? h : max_hits;
            }
        }
    }
    g.flush_stages = wg_chain(cg) / (max_hits * g.Q / 2);
    if (g.flush_stages < 1)
        g.flush_stages = 1;
    g.kd_a16 = g.X * g.r8;
    // offsets of a stage's items are 32 bits, in elements (a lane's own channel of four is added
    // to the base pointer): 16 filters of 2^28 cells in one role
    if ((cgp - 1) / 4 * 4 * (double) cg.xs_c + (kdg - 1) * (double) cg.xs[0] + g.X * (double) cg.xs[1] + 4.0 * PW >= 4294967296.0
        || (kg - 1) / 4 * 4 * (double) cg.ys_c + B * (double) cg.ys[1] + 4.0 * PW >= 4294967296.0)
        return false;
    // shared memory; 16 bytes behind every 128-byte multiple of cells keep the
    // converters' stores (eight cells of a row at a time) on different banks
    const int planes = ring ? 1 : kdg; // of x that a stage brings
    g.ring = ring;
    g.xrows = planes * g.X * g.r8;
    g.yrows = B * g.n8;
    g.lbo_x = g.xrows * 16 + 16;
    g.lbo_y = g.yrows * 16 + 16;
    g.y_off = (g.Q * g.lbo_x + 127) / 128 * 128;
    g.stage_bytes = g.y_off + (g.Q * g.lbo_y + 127) / 128 * 128;
    g.cq = (cgp + 3) / 4;
    g.kq = (kg + 3) / 4;
    g.qg = (g.Q + 7) / 8;
    g.items_x = planes * g.X * g.cq * g.qg;
    g.items_y = B * g.kq * g.qg;
    const int tail = WG_MAX_TILES * (int) sizeof(WgTile) + (g.items_x + g.items_y) * 16 + 256 + 2048 + 128;
    const int room = 226 * 1024 - tail, dump = g.kd_cols * 512;
    g.nstages = room / g.stage_bytes < WG_MAX_STAGES ? room / g.stage_bytes : WG_MAX_STAGES;
    if (g.nstages < (ring ? kdg + 1 : 2) || dump > room || g.lbo_x >= 1 << 18 || g.lbo_y >= 1 << 18)
        return false;
    const int body = g.nstages * g.stage_bytes > dump ? g.nstages * g.stage_bytes : dump;
    g.so_tiles = (body + 127) / 128 * 128;
    g.so_items = g.so_tiles + WG_MAX_TILES * (int) sizeof(WgTile);
    g.so_bars = g.so_items + (g.items_x + g.items_y) * 16;
    // an instruction reads 128 rows from a tile's first one, used or not: the slack keeps that inside
    g.smem = g.so_bars + 256 + 2048 + 128;
    g.hblocks = (cg.out[1] + B - 1) / B;
    g.wchunks = (cg.out[2] + PW - 1) / PW;
    g.stages = (long long) cg.n * cg.out[0] * g.hblocks * g.wchunks;
    if (g.stages >= (1ll << 31))
        return false;
    g.parts = g.roles < sms ? sms / g.roles : 1;
    if (g.parts > g.stages)
        g.parts = (int) g.stages;
    // clocks of a stage: the tensor pipe, the converters' instructions, their latency
    const double pipe = kdg * mma * (g.Q / 2) * 1.1 + 200.0;
    const int nv = 3 * cg.stride[2] + kwg;
    const double ix = 60.0 + 6.0 * nv + 4.0 * kwg, iy = 70.0;
    const double instr = (g.items_x * ix + g.items_y * iy) / 4.0 * 1.3;
    // warps for x and dy: the longer of their chains of item pairs, and where several
    // splits have the same longest chain, the one whose warps are busy alike on average
    double lat = 1e30, best = 1e30;
    for (int wx = 1; wx < WG_CONV; ++wx)
    {
        const int wy = WG_CONV - wx;
        const double lx = 200.0 + 4.0 * ix, ly = 200.0 + 4.0 * iy;
        const double px = (double) ((g.items_x + 2 * wx - 1) / (2 * wx)) * lx,
                     py = (double) ((g.items_y + 2 * wy - 1) / (2 * wy)) * ly;
        const double ax = g.items_x * lx / (2.0 * wx), ay = g.items_y * ly / (2.0 * wy);
        const double m = px > py ? px : py, score = m + 0.3 * (ax > ay ? ax : ay);
        if (score < best)
            best = score, lat = m, g.warps_x = wx;
    }
    // The terms' weights are a fit to the times of 1200 layouts of 33 layers (8 % rms; the layout
    // that it picked of a layer was 1 % slower than the best of it, with all weights 1 it was 9 %):
    // pipe and converters overlap in part, stages narrower than 32 positions fetch parts of lines,
    // a walk's lead steps bring a plane each, a piece of eight columns costs a flush 280. The fit is older
    // than the converters' lanes along the row. Of the best walk and the best plain layout of 61 layers,
    // both timed with those, it picks one that is 0.7 % slower than the other (geometric mean; 22 % at worst,
    // 6 -> 32 on 90 x 160 x 16); 8 -> 24 on 2 x 67 x 83 x 101 takes 285 us and would take 256 as a walk.
    const double feed = std::max(instr, lat);
    const double narrow = 1.0 + 0.285 * std::max(0, 32 - PW) / 32.0;
    const double per = (1.2 * std::max(pipe, feed) + 0.64 * std::min(pipe, feed) + 530.0) * narrow;
    const double waves = (double) ((g.roles + sms - 1) / sms);
    const double n = (double) ((g.stages + g.parts - 1) / g.parts);
    const double lead = ring ? 0.7 * (kdg - 1) * (n / cg.out[0] + 1.0) : 0.0;
    const double harvest = kdg * (g.nblocks * g.n8 * 35.0 + kg * cgp * kwg * 5.5);
    const double flush = n / g.flush_stages * (kdg * g.nblocks * (g.kgp / 8)) * 280.0;
    *cost = g.nkw * (waves * ((n + lead + 0.3) * per + flush + harvest) + 24000.0);
    return true;
}

} // namespace

// Geometry of the tensor-core backward filter: x is the forward input window,
// dy the forward output window.
bool wg_geom(const ConvGeom& cg, int math_mode, int sms, WgGeom* out)
{
    if (math_mode == DCB_MATH_FP32_SIMT)
        return false;
    for (int i = 0; i < 3; ++i)
        if (cg.stride[i] < 1 || cg.stride[i] > 2 || cg.dil[i] != 1 || cg.pad[i] > cg.f[i] - 1 || cg.f[i] > 16)
            return false;
    if ((long long) cg.n * cg.out[0] * cg.out[1] * cg.out[2] == 0 || cg.c == 0 || cg.k == 0
        || cg.f[0] * cg.f[1] * cg.f[2] > 128)
        return false;
    WgGeom g, best;
    std::memset(&g, 0, sizeof(g));
    g.n = cg.n, g.c = cg.c, g.k = cg.k;
    for (int i = 0; i < 3; ++i)
    {
        g.in[i] = cg.in[i], g.out[i] = cg.out[i], g.f[i] = cg.f[i], g.pad[i] = cg.pad[i], g.stride[i] = cg.stride[i];
        g.xs[i] = cg.xs[i], g.ys[i] = cg.ys[i];
    }
    g.xs_n = cg.xs_n, g.xs_c = cg.xs_c, g.ys_n = cg.ys_n, g.ys_c = cg.ys_c;
    double best_cost = -1;
    for (int kwg : {1, 3, 5})
    {
        if (kwg > cg.f[2] && kwg > 1 && kwg - cg.f[2] > 1)
            continue;
        int last_c = 0;
        for (int nc = 1; nc <= 64 && nc <= cg.c; ++nc)
        {
            const int cgp = (cg.c + nc - 1) / nc;
            if (cgp == last_c || 2 * cgp * kwg > 128)
                continue;
            last_c = cgp;
            for (int kdg = cg.f[0]; kdg >= 1; kdg = kdg == 1 ? 0 : (kdg + 1) / 2)
            {
                int last_k = 0;
                for (int nk = 1; nk <= 16 && nk <= cg.k; ++nk)
                {
                    const int kg = (cg.k + nk - 1) / nk;
                    if (kg == last_k)
                        continue;
                    last_k = kg;
                    for (int B : {1, 2, 3, 4, 6, 8, 12})
                    {
                        if (B > 1 && B > cg.out[1])
                            break;
                        for (int chunks = 1; chunks <= (cg.out[2] + 7) / 8; ++chunks)
                        {
                            const int pw = ((cg.out[2] + chunks - 1) / chunks + 7) / 8 * 8;
                            if (pw > 64)
                            {
                                chunks = (cg.out[2] + 63) / 64 - 1;
                                continue;
                            }
                            if (pw < 16 && chunks > 1)
                                break;
                            double cost;
                            // all planes kd in one role and unit stride along D: a walk along D converts a
                            // plane of x once, not once per kd, and needs kdg - 1 steps to begin with
                            // (256 x 256 x D: D = 8 72 us, 68 without a walk; D = 16 103 and 113)
                            for (int walk = 0; walk < 2; ++walk)
                                if ((walk == 0 || (kdg > 1 && kdg == cg.f[0] && cg.stride[0] == 1 && cg.out[0] >= 4))
                                    && wg_layout(cg, &g, cgp, kwg, kdg, kg, B, pw, walk == 1, sms, &cost)
                                    && (best_cost < 0 || cost < best_cost))
                                    best_cost = cost, best = g;
                            if (pw <= 16)
                                break;
                            // the next width that is a smaller multiple of 8
                            const int next = pw - 8;
                            chunks = (cg.out[2] + next - 1) / next - 1;
                        }
                    }
                }
            }
        }
    }
    if (best_cost < 0)
        return false;
    *out = best;
    return true;
}

} // namespace dcb
