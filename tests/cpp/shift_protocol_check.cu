// The shift kernel's barriers between issuers and epilogue, in the layouts that the planner gives: every
// warp's waits and arrivals in program order, run in orders where one of them is as far behind the others as it can
// be.  Prints how many passes were looked at, how many of them open and close a plane in one step with
// several rows a column, and in how many an arrival or a wait meets another use of its block than its own,
// or nobody can go on.  Host code only; links against the library.
#include "conv_tc_shift_plan.cuh"

#include <cstdio>
#include <cstring>
#include <deque>
#include <random>

using namespace dcb;

struct Op
{
    bool wait, empty; // else an arrival; on ev_empty, else ev_full
    int block, use;
};

struct Barrier
{
    int count, pending, phase = 0;
};

constexpr unsigned GRID = 148;

static std::vector<Op> issuer(const ShGeom& g, int w)
{
    std::vector<Op> ops;
    std::vector<int> reported((size_t) g.th * g.ns, 0);
    const int ahead = sh_reports_ahead(g);
    int skip = w, first_slot = 0, first_lap = 0, last_slot = 0;
    for (unsigned unit = 0; unit < g.units; unit += GRID)
    {
        const ShUnit u = sh_unit(g, unit);
        const int nq = (u.nz - g.fs) / g.st_s + 1;
        int opened = 0, closed = 0;
        for (int z = 0; z < u.nz; ++z)
        {
            const bool opens = opened * g.st_s == z && opened < nq, closes = closed * g.st_s + g.fs - 1 == z;
            const bool real = z >= u.z_lo && z < u.z_hi;
            int j_open = opens && first_lap > 0 ? 0 : g.th;
            auto open = [&]() { ops.push_back({true, true, j_open++ * g.ns + first_slot, first_lap - 1}); };
            for (int grp = 0; grp < g.cgroups; ++grp)
            {
                int j_close = closes && grp + 1 == g.cgroups ? 0 : g.th;
                auto report = [&]() {
                    const int b = j_close++ * g.ns + last_slot;
                    ops.push_back({false, false, b, reported[(size_t) b]++});
                };
                int i = real ? u.i_lo + skip : g.rows;
                if (real)
                    for (skip -= u.i_hi - u.i_lo; skip < 0;)
                        skip += SH_ISS;
                for (; real && i < u.i_hi; i += SH_ISS)
                {
                    while (j_open < g.th && j_open * g.st_r <= i)
                        open();
                    while (j_close < g.th && j_close * g.st_r + g.fr - 1 < i + ahead)
                        report();
                }
                while (grp == 0 && j_open < g.th)
                    open();
                while (j_close < g.th)
                    report();
            }
            if (opens)
            {
                ++opened;
                if (++first_slot == g.ns)
                    first_slot = 0, ++first_lap;
            }
            if (closes)
            {
                ++closed;
                last_slot = (last_slot + 1) % g.ns;
            }
        }
    }
    return ops;
}

static std::vector<Op> epilogue(const ShGeom& g, int warp)
{
    std::vector<Op> ops;
    const bool shared = sh_shared_drain(g);
    const int team = warp >> 2, teams = std::min(SH_EPI / 4, g.th * g.ns);
    int slot = 0, lap = 0, j = shared ? 0 : team < teams ? team : 0x40000000;
    for (unsigned unit = 0; unit < g.units; unit += GRID)
    {
        const ShUnit u = sh_unit(g, unit);
        for (int qi = 0; qi < (u.nz - g.fs) / g.st_s + 1; ++qi)
        {
            for (; j < g.th; j += shared ? 1 : teams)
            {
                ops.push_back({true, false, j * g.ns + slot, lap});
                ops.push_back({false, true, j * g.ns + slot, lap});
            }
            j -= g.th;
            if (++slot == g.ns)
                slot = 0, ++lap;
        }
    }
    return ops;
}

// behind: the actor that moves only when no other can (-1: at random)
static bool run(const ShGeom& g, const std::vector<std::vector<Op>>& programs, int behind, unsigned seed)
{
    const int blocks = g.th * g.ns, actors = (int) programs.size() + SH_ISS; // the issuers' commits arrive later, in order
    std::vector<Barrier> full((size_t) blocks, {SH_ISS, SH_ISS}), empty((size_t) blocks, {0, 0});
    for (Barrier& b : empty)
        b.count = b.pending = sh_shared_drain(g) ? SH_EPI : 4;
    std::vector<size_t> at(programs.size(), 0);
    std::vector<std::deque<Op>> commits(SH_ISS);
    bool good = true;
    auto arrive = [&](const Op& o) {
        Barrier& b = (o.empty ? empty : full)[(size_t) o.block];
        good = good && b.phase == o.use;
        if (--b.pending == 0)
            b.pending = b.count, ++b.phase;
    };
    auto step = [&](int a) {
        if (a >= (int) programs.size())
        {
            auto& q = commits[(size_t) (a - (int) programs.size())];
            if (q.empty())
                return false;
            arrive(q.front());
            q.pop_front();
            return true;
        }
        if (at[(size_t) a] == programs[(size_t) a].size())
            return false;
        const Op o = programs[(size_t) a][at[(size_t) a]];
        if (o.wait)
        {
            const Barrier& b = (o.empty ? empty : full)[(size_t) o.block];
            good = good && b.phase <= o.use + 1;
            if (((b.phase ^ o.use) & 1) == 0)
                return false;
            good = good && b.phase == o.use + 1;
        }
        else if (a < SH_ISS)
            commits[(size_t) a].push_back(o);
        else
            arrive(o);
        ++at[(size_t) a];
        return true;
    };
    std::mt19937 rng(seed);
    for (bool moved = true; moved && good;)
    {
        moved = false;
        const int from = (int) (rng() % (unsigned) actors);
        for (int k = 0; k < actors && good; ++k)
        {
            const int a = (from + k) % actors;
            for (unsigned n = a == behind ? 0 : behind < 0 ? rng() % 8 : 1000; n > 0 && step(a); --n)
                moved = true;
        }
        if (!moved && good)
            for (int a = 0; a < actors && !moved; ++a)
                moved = step(behind >= 0 && a == 0 ? behind : a);
    }
    for (size_t a = 0; a < programs.size(); ++a)
        good = good && at[a] == programs[a].size();
    return good;
}

int main()
{
    int passes = 0, same = 0, bad = 0;
    struct Layer
    {
        int n, c, k, in[3], f[3], s;
    };
    for (const Layer& l : {Layer{3, 4, 3, {56, 51, 132}, {1, 1, 1}, 1}, {1, 16, 16, {20, 60, 70}, {1, 1, 1}, 1}, {1, 8, 32, {40, 64, 64}, {1, 2, 2}, 1},
                           {1, 8, 8, {40, 64, 64}, {1, 3, 3}, 1}, {1, 8, 8, {40, 64, 64}, {1, 3, 3}, 2}, {2, 16, 8, {30, 40, 50}, {2, 2, 2}, 2},
                           {1, 4, 16, {64, 64, 64}, {1, 1, 1}, 2}, {1, 4, 16, {32, 64, 130}, {3, 3, 3}, 1}, {1, 16, 32, {64, 64, 64}, {3, 3, 3}, 2},
                           {1, 8, 16, {40, 60, 70}, {3, 1, 1}, 1}, {1, 8, 16, {40, 60, 70}, {2, 2, 2}, 1}, {1, 24, 28, {20, 50, 132}, {3, 3, 3}, 1},
                           {1, 8, 8, {40, 64, 64}, {1, 5, 5}, 1}, {2, 8, 24, {40, 83, 101}, {3, 3, 3}, 1}, {1, 32, 32, {0, 200, 64}, {1, 5, 5}, 1}})
        for (int tr = 0; tr < 2; ++tr)
            for (int math : {DCB_MATH_FP32, DCB_MATH_TF32, DCB_MATH_BF16})
            {
                ConvGeom g;
                std::memset(&g, 0, sizeof(g));
                g.n = l.n, g.c = l.c, g.k = l.k;
                for (int i = 0; i < 3; ++i)
                {
                    g.in[i] = std::max(1, l.in[i]), g.f[i] = l.f[i], g.pad[i] = (l.f[i] - 1) / 2, g.stride[i] = l.in[i] ? l.s : 1, g.dil[i] = 1;
                    g.out[i] = (g.in[i] + 2 * g.pad[i] - g.f[i]) / g.stride[i] + 1;
                }
                g.xs[2] = g.ys[2] = 1;
                for (int i = 1; i >= 0; --i)
                    g.xs[i] = g.xs[i + 1] * g.in[i + 1], g.ys[i] = g.ys[i + 1] * g.out[i + 1];
                g.xs_c = g.xs[0] * g.in[0], g.xs_n = g.xs_c * g.c;
                g.ys_c = g.ys[0] * g.out[0], g.ys_n = g.ys_c * g.k;
                ShTables t;
                if (!ShBuilder(g, tr == 1, math, (int) GRID).build(&t))
                    continue;
                std::vector<std::vector<Op>> programs;
                for (int w = 0; w < SH_ISS; ++w)
                    programs.push_back(issuer(t.g, w));
                for (int w = 0; w < SH_EPI; ++w)
                    programs.push_back(epilogue(t.g, w));
                bool good = true;
                for (int behind = -6; behind < (int) programs.size() + SH_ISS && good; ++behind)
                    good = run(t.g, programs, behind, (unsigned) (behind + 7));
                ++passes;
                same += t.g.fs == 1 && t.g.th > 1;
                bad += !good;
            }
    std::printf("%d %d %d\n", passes, same, bad);
    return 0;
}
