// Shift kernel: how a convolution is dealt out, and the kernel's tables.  Host code
// only: needs no device.
#include "conv_tc_shift_plan.cuh"

namespace dcb
{

namespace
{

constexpr int SH_SMEM_MAX = 226 * 1024;
constexpr int SH_FOREIGN = -2; // column of a block that a row does not add to

// The tensor pipe adds by truncation: a chain of n updates is off by about 2e-8 n of the
// result, where the sums have a mean.  No chain of leading products is longer than this;
// a layer that would need one takes the CUDA-core kernels.
constexpr int SH_CHAIN_MAX = 96;
// ... and most layers stay below this: 1e-6, as 3xTF32 products with one chain per
// channel group.
constexpr int SH_CHAIN_LOOSE = 60;

int align_up(int v, int a)
{
    return (v + a - 1) / a * a;
}

} // namespace

std::vector<int> ShBuilder::row_code(const ShGeom& g, int phase, int i, int ew) const
{
    std::vector<int> code((size_t) TC_TMEM_COLS, SH_FOREIGN);
    for (int c = 0; c < (int) TC_TMEM_COLS; ++c)
    {
        const int in_row = c % g.rowst;
        if (c >= g.set_off || in_row >= g.ns * g.blk)
            code[(size_t) c] = -1; // nobody's
    }
    for (int m = 0;; ++m)
    {
        const int ts = phase % g.st_s + m * g.st_s;
        if (ts >= g.fs)
            break;
        const int slot = ((phase / g.st_s - m) % g.ns + g.ns) % g.ns;
        for (int j = 0; j < g.th; ++j)
        {
            const int tr = i - j * g.st_r;
            if (tr < 0 || tr >= g.fr)
                continue;
            for (int c = 0; c < g.blk; ++c)
                code[(size_t) (ew * g.woff + j * g.rowst + slot * g.blk + c)] = -1; // open: may be covered with zeros
            for (int es = 0; es < g.e_s; ++es)
                for (int er = 0; er < g.e_r; ++er)
                {
                    const int ks = m_s.k(ts, es), kr = m_r.k(tr, er);
                    if (ks < 0 || kr < 0)
                        continue;
                    const int base = (m_flat ? ks : ks * m_cg.f[1] + kr) * m_cg.f[2];
                    const int col = ew * g.woff + j * g.rowst + slot * g.blk + (es * g.e_r + er) * g.nb;
                    for (int ko = 0; ko < g.kcols; ++ko)
                        code[(size_t) (col + ko)] = ko << 16 | base;
                }
        }
    }
    return code;
}

// Column ranges (multiples of 16, at most 256 wide) that cover the used columns
// at the least cost.  Unused columns of open blocks may be covered with zeros,
// blocks that the row does not add to may not.
std::vector<std::pair<int, int>> ShBuilder::ranges(const std::vector<int>& code) const
{
    std::vector<int> u, foreign((size_t) code.size() / 16 + 1, 0); // used 16-column pieces; foreign ones before a piece
    for (int b = 0; b < (int) code.size() / 16; ++b)
    {
        bool used = false, other = false;
        for (int c = 0; c < 16; ++c)
        {
            used = used || code[(size_t) (b * 16 + c)] >= 0;
            other = other || code[(size_t) (b * 16 + c)] == SH_FOREIGN;
        }
        if (used)
            u.push_back(b);
        foreign[(size_t) b + 1] = foreign[(size_t) b] + (other ? 1 : 0);
    }
    const int m = (int) u.size();
    std::vector<double> best((size_t) m + 1, 1e30);
    std::vector<int> from((size_t) m + 1, 0);
    best[0] = 0;
    for (int k = 1; k <= m; ++k)
        for (int l = k - 1; l >= 0; --l)
        {
            const int n = 16 * (u[(size_t) k - 1] - u[(size_t) l] + 1);
            if (n > 256 || foreign[(size_t) u[(size_t) k - 1] + 1] != foreign[(size_t) u[(size_t) l]])
                break;
            const double c = best[(size_t) l] + sh_mma_cost(n);
            if (c < best[(size_t) k])
                best[(size_t) k] = c, from[(size_t) k] = l;
        }
    std::vector<std::pair<int, int>> r;
    for (int k = m; k > 0; k = from[(size_t) k])
    {
        const int a = u[(size_t) from[(size_t) k]];
        r.push_back({a * 16, 16 * (u[(size_t) k - 1] - a + 1)});
    }
    std::reverse(r.begin(), r.end());
    return best[(size_t) m] < 1e30 ? r : std::vector<std::pair<int, int>>();
}

// The k-steps of a staged row, per cell parity of the output row (ew) and per
// accumulator set, and the filter-image cells they read.
void ShBuilder::make_steps(ShTables* T, int J, std::vector<std::vector<std::vector<ShStep>>>* steps,
                           std::vector<std::vector<ShChunk>>* chunks) const
{
    const ShGeom& g = T->g;
    struct Prod
    {
        int pa, pb;
    };
    std::vector<Prod> prods = {{0, 0}};
    if (m_parts == 2)
        prods = {{0, 0}, {1, 0}, {0, 1}};
    if (m_parts == 3)
        prods = {{0, 0}, {1, 0}, {2, 0}, {0, 1}, {1, 1}, {0, 2}};
    steps->assign((size_t) g.e_w, std::vector<std::vector<ShStep>>((size_t) g.nsets));
    chunks->assign((size_t) g.e_w, {});
    for (int ew = 0; ew < g.e_w; ++ew)
    {
        struct Tap
        {
            int off, kw;
        };
        std::vector<Tap> taps; // offset inside a cell's planes, filter tap
        for (int t = 0; t < m_w.taps; ++t)
            if (m_w.k(t, ew) >= 0)
                taps.push_back({(t % m_w.st) * g.pt + t / m_w.st, m_w.k(t, ew)});
        const int lead = g.nsets - (m_parts > 1 && g.nsets > 1 ? 1 : 0); // sets of the leading products
        std::vector<ShChunk>& ck = (*chunks)[(size_t) ew];
        auto a_of = [&](int p, int j, const Tap& t) { return (p * J + j) * m_w.st * g.pt + t.off; };
        struct Item
        {
            int a, pa, j, tap;
            ShChunk c;
        };
        for (int set = 0; set < g.nsets; ++set)
        {
            std::vector<ShStep>& out = (*steps)[(size_t) ew][(size_t) set];
            auto add = [&](int a0, const ShChunk& c0, int a1, const ShChunk& c1) {
                int at = -1;
                for (size_t i = 0; i + 1 < ck.size(); ++i)
                    if (ck[i] == c0 && ck[i + 1] == c1)
                    {
                        at = (int) i;
                        break;
                    }
                if (at < 0)
                {
                    at = (int) ck.size();
                    ck.push_back(c0);
                    ck.push_back(c1);
                }
                out.push_back({a0, a1, at});
            };
            std::vector<Item> left;
            for (const Prod& pr : prods)
            {
                std::vector<Item> list;
                for (int j = 0; j < J; ++j)
                    for (size_t t = 0; t < taps.size(); ++t)
                    {
                        int want = 0;
                        if (m_parts > 1 && pr.pa + pr.pb > 0)
                            want = g.nsets - 1;
                        else
                            want = (int) ((j * taps.size() + t) * (size_t) lead / (J * taps.size()));
                        if (want == set)
                            list.push_back({a_of(pr.pa, j, taps[t]), pr.pa, j, (int) t,
                                            {pr.pb, taps[t].kw, j * m_ch}});
                    }
                std::sort(list.begin(), list.end(), [](const Item& x, const Item& y) { return x.a < y.a; });
                size_t i = 0;
                for (; i + 1 < list.size(); i += 2)
                    add(list[i].a, list[i].c, list[i + 1].a, list[i + 1].c);
                if (i < list.size())
                    left.push_back(list[i]);
            }
            std::stable_sort(left.begin(), left.end(), [](const Item& x, const Item& y) { return x.a < y.a; });
            std::vector<char> used(left.size(), 0);
            const ShChunk zero = {-1, 0, 0};
            for (size_t i = 0; i < left.size(); ++i)
            {
                if (used[i])
                    continue;
                size_t k = i + 1;
                while (k < left.size() && (used[k] || left[k].a == left[i].a))
                    ++k;
                if (k < left.size())
                {
                    used[k] = 1;
                    add(left[i].a, left[i].c, left[k].a, left[k].c);
                    continue;
                }
                // alone: beside it, against zeros, a cell of the same output's own taps
                const Item& it = left[i];
                if (it.tap > 0)
                    add(a_of(it.pa, it.j, taps[0]) < it.a ? a_of(it.pa, it.j, taps[0]) : it.a - 1, zero, it.a, it.c);
                else if (taps.size() > 1 && a_of(it.pa, it.j, taps[1]) > it.a)
                    add(it.a, it.c, a_of(it.pa, it.j, taps[1]), zero);
                else
                    add(it.a, it.c, it.a + 1, zero);
            }
        }
    }
}

bool ShBuilder::layout(const Try& t, ShTables* T) const
{
    ShGeom& g = T->g;
    std::memset(&g, 0, sizeof(g));
    const ConvGeom& cg = m_cg;
    const long long* ss = m_tr ? cg.ys : cg.xs;
    const long long* os = m_tr ? cg.xs : cg.ys;
    g.n = cg.n;
    g.cin = m_cin, g.kout = m_kout;
    g.in_s = m_s.in, g.in_r = m_r.in, g.in_w = m_w.in;
    g.q_s = m_s.q, g.q_r = m_r.q, g.q_w = m_w.q;
    g.o_s = m_s.o, g.o_r = m_r.o, g.o_w = m_w.o;
    g.xs_n = m_tr ? cg.ys_n : cg.xs_n, g.xs_c = m_tr ? cg.ys_c : cg.xs_c;
    g.ys_n = m_tr ? cg.xs_n : cg.ys_n, g.ys_c = m_tr ? cg.xs_c : cg.ys_c;
    g.xs_s = ss[m_flat ? 1 : 0], g.xs_r = m_flat ? 0 : ss[1];
    g.ys_s = os[m_flat ? 1 : 0], g.ys_r = m_flat ? 0 : os[1];
    g.st_s = m_s.st, g.st_r = m_r.st, g.st_w = m_w.st;
    g.e_s = m_s.e, g.e_r = m_r.e, g.e_w = m_w.e;
    g.fs = m_s.taps, g.fr = m_r.taps;
    g.pad_s = m_s.pad, g.pad_r = m_r.pad, g.pad_w = m_w.pad;
    g.kgroups = t.kg;
    g.kcols = (m_kout + t.kg - 1) / t.kg;
    if ((g.kgroups - 1) * g.kcols >= m_kout)
        return false;
    g.nb = g.kcols <= 4 ? 4 : (g.kcols <= 8 ? 8 : (g.kcols <= 16 ? 16 : align_up(g.kcols, 4)));
    g.th = t.th;
    g.rows = (g.th - 1) * g.st_r + g.fr;
    g.ns = t.ns;
    g.nph = g.ns * g.st_s;
    g.nsets = t.nsets;
    g.blk = g.nb * g.e_s * g.e_r;
    // Instructions update whole multiples of 16 columns, also with zeros, and an
    // update with zeros of a block that the epilogue is draining would bring its old
    // values back.  Rows of blocks start on such multiples; the plane slots of a row
    // have to as well, unless every staged plane adds to all of them.
    if (m_flat || m_s.st > 1)
        g.blk = align_up(g.blk, 16);
    g.rowst = align_up(g.ns * g.blk, 16);
    g.woff = g.th * g.rowst;
    g.set_off = g.e_w * g.woff;
    if (sh_columns(g) > (int) TC_TMEM_COLS || g.th * g.ns > SH_MAX_BLOCKS)
        return false;
    const int cells = (m_cin + m_ch - 1) / m_ch;
    const int J = (cells + t.cgroups - 1) / t.cgroups;
    if ((t.cgroups - 1) * J >= cells)
        return false;
    g.cgroups = t.cgroups;
    g.cpg = J * m_ch;
    const int reach = (m_w.taps - 1) / m_w.st; // positions to the right of an output's own
    if (t.wt > 0)
    {
        // rows, or equal parts of them, several sub-columns side by side
        const int segs_left = m_flat ? t.nseg : (g.q_r + g.th - 1) / g.th;
        g.tile_w = (g.q_w + t.wt - 1) / t.wt;
        g.tiles_w = (g.q_w + g.tile_w - 1) / g.tile_w;
        g.npack = std::min(packed(g.tile_w), segs_left);
    }
    else
    {
        g.npack = 1;
        g.tiles_w = (g.q_w + TC_M - 1) / TC_M;
        g.tile_w = std::min(TC_M, align_up((g.q_w + g.tiles_w - 1) / g.tiles_w, 32));
        g.tiles_w = (g.q_w + g.tile_w - 1) / g.tile_w;
    }
    // what the row's outputs read: a tile is whole warps, but what lies behind a row that is its
    // only one needs no converter item (backward data of 8 -> 24 on 2 x 67 x 83 x 101: four items
    // instead of five, three teams of converters instead of one, 245 -> 175 us)
    T->per = (g.tiles_w == 1 ? std::min(g.tile_w, g.q_w) : g.tile_w) + reach;
    const int used = g.npack * T->per;
    g.pt = std::max(TC_M + reach, g.npack * (g.tile_w + reach)) + 1;
    const int npb = (used + 31) / 32;
    g.ipr = g.st_w * npb;
    if (g.ipr > SH_MAX_ITEMS)
        return false;
    g.a_slot16 = m_parts * J * g.st_w * g.pt;
    g.seglen = (g.q_s + t.nseg - 1) / t.nseg;
    g.nsegs = (g.q_s + g.seglen - 1) / g.seglen;
    g.hblks = (g.q_r + g.th - 1) / g.th;
    if (g.npack > 1 && m_flat)
    {
        g.pack_s = g.seglen;
        g.nsegs = (g.nsegs + g.npack - 1) / g.npack;
    }
    else if (g.npack > 1)
    {
        g.pack_r = g.th;
        g.hblks = (g.hblks + g.npack - 1) / g.npack;
    }
    const long long units = (long long) g.n * g.kgroups * g.tiles_w * g.hblks * g.nsegs;
    if (units >= (1ll << 31))
        return false;
    g.units = (unsigned) units;
    g.rnd_add = m_bf16 ? 0x8000u : 0x1000u;
    g.rnd_mask = m_bf16 ? 0xffff0000u : 0xffffe000u;
    // a lane's offsets from a row's base pointer are 32 bits, in bytes: the sub-columns' distance,
    // the row and, unless they lie too far apart, three channel strides
    const double subs = g.npack > 1 ? g.npack * ((double) g.pack_s * g.st_s * g.xs_s + (double) g.pack_r * g.st_r * g.xs_r) : 0.0,
                 reach_bytes = 4.0 * (subs + 2.0 * g.in_w);
    if (reach_bytes >= 2147483648.0)
        return false;
    T->wide = reach_bytes + 12.0 * g.xs_c >= 2147483648.0;
    T->kind = m_kind, T->parts = m_parts, T->c_of_cell = m_ch;
    const int taps = cg.f[0] * cg.f[1] * cg.f[2];
    T->w_ko = m_tr ? taps : (long long) cg.c * taps;
    T->w_ci = m_tr ? (long long) cg.c * taps : taps;
    ShExact& e = T->exact;
    std::memset(&e, 0, sizeof(e));
    e.transposed = m_tr, e.one_pass = m_parts == 1;
    e.w_ko = T->w_ko, e.w_ci = T->w_ci;
    for (int d = 0; d < 3; ++d)
    {
        const int i = m_flat && d < 2 ? 1 - d : d; // an image is swept along H
        e.f[d] = cg.f[i], e.stride[d] = cg.stride[i], e.pad[d] = cg.pad[i];
    }
    return true;
}

// Sub-columns of w outputs that fit the 128 lanes side by side.
int ShBuilder::packed(int w) const
{
    const int reach = (m_w.taps - 1) / m_w.st;
    return w > TC_M ? 0 : (TC_M - w) / (w + reach) + 1;
}

// Parts that rows may be cut in to lie side by side (0: whole tiles of 32, one beside no other).
// Rows of up to 63 outputs fit whole, several of them.  A row of 64 has room for one (64 + 66
// positions) and one of 132 is two tiles of 96, half of the lanes of either idle: 16 outputs of seven
// rows fill 112 lanes, 22 of five 110.  Such parts are stored by registers and read their
// neighbours' cells again, so they are only tried where they fill a good deal more of the lanes.
// us, forward and backward data: 32 -> 32 on 2 x 24 x 40 x 64 151 -> 82 and 156 -> 82, 24 -> 28 on 40 x 100 x 132
// 541 -> 312 and 453 -> 258, 12 -> 20 on 50 x 90 x 177 132 -> 101 and 151 -> 126, 16 -> 24 with stride 2
// on 90 x 90 x 160 backward data 77 -> 58. Of 260 layers drawn over the range, 2 % less time for all together forward
// and 3 % backward; the worst is 8 -> 32 with stride 2 on 4 images of 40 x 200, 10.2 -> 10.8. (The shares of the
// lanes below which parts are not tried are set by hand, to keep the search short; the clocks decide.)
std::vector<int> ShBuilder::row_parts() const
{
    if (packed(m_w.q) >= 2)
        return {1};
    const int tiles = (m_w.q + TC_M - 1) / TC_M;
    const double whole = (double) m_w.q / (tiles * TC_M);
    double most = 0;
    std::vector<std::pair<int, double>> fill;
    for (int parts = tiles + 1; parts <= 8 * tiles && parts <= m_w.q / 8; ++parts)
    {
        const int w = (m_w.q + parts - 1) / parts, n = packed(w);
        if (n < 2 || (m_w.q + w - 1) / w != parts)
            continue;
        const double f = (double) n * m_w.q / (parts * TC_M);
        fill.push_back({parts, f});
        most = std::max(most, f);
    }
    std::vector<int> r = {0};
    // the widest that come close to the best
    for (const auto& f : fill)
        if (r.size() < 3 && f.second > 1.15 * whole && f.second > (r.size() == 1 ? 0.85 : 0.97) * most)
            r.push_back(f.first);
    return r;
}

// Fills in the tables; false when something does not fit shared memory.
bool ShBuilder::finish(const Try& t, ShTables* T) const
{
    ShGeom& g = T->g;
    const int J = g.cpg / m_ch;
    std::vector<std::vector<std::vector<ShStep>>> steps;
    std::vector<std::vector<ShChunk>> chunks;
    make_steps(T, J, &steps, &chunks);

    // accumulator ranges of every (phase, row), widest first so that narrower
    // ones (rows at the edge of a column) are found inside an existing image
    struct Range
    {
        int phase, i, ew, col, n;
        std::vector<int> code;
        int image, at;
    };
    std::vector<Range> all;
    for (int ph = 0; ph < g.nph; ++ph)
        for (int i = 0; i < g.rows; ++i)
            for (int ew = 0; ew < g.e_w; ++ew)
            {
                const std::vector<int> code = row_code(g, ph, i, ew);
                const auto rs = ranges(code);
                if (rs.empty() && *std::max_element(code.begin(), code.end()) >= 0)
                    return false; // a used piece that another block shares
                for (const auto& r : rs)
                    all.push_back({ph, i, ew, r.first, r.second,
                                   std::vector<int>(code.begin() + r.first, code.begin() + r.first + r.second), -1, 0});
            }
    std::vector<int> order(all.size());
    for (size_t i = 0; i < order.size(); ++i)
        order[i] = (int) i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return all[(size_t) a].n > all[(size_t) b].n; });

    std::vector<ShImage> images;
    std::vector<int> set_off, set_size;
    int total16 = 0;
    auto place = [&](bool stream) {
        images.clear();
        for (int idx : order)
        {
            Range& r = all[(size_t) idx];
            r.image = -1;
            for (size_t m = 0; m < images.size() && r.image < 0; ++m)
            {
                const ShImage& im = images[m];
                if (im.ew != r.ew || (stream && im.set != r.phase))
                    continue;
                for (int at = 0; at + r.n <= (int) im.code.size(); at += 16)
                    if (std::equal(r.code.begin(), r.code.end(), im.code.begin() + at))
                    {
                        r.image = (int) m, r.at = at;
                        break;
                    }
            }
            if (r.image < 0)
            {
                r.image = (int) images.size(), r.at = 0;
                images.push_back({r.ew, r.code, stream ? r.phase : 0, 0});
            }
        }
        const int nsets = stream ? g.nph : 1;
        set_off.assign((size_t) nsets, 0);
        set_size.assign((size_t) nsets, 0);
        total16 = 0;
        for (int s = 0; s < nsets; ++s)
        {
            set_off[(size_t) s] = total16;
            for (ShImage& im : images)
                if (im.set == s)
                {
                    im.off16 = total16 - set_off[(size_t) s];
                    total16 += (int) (im.code.size() * chunks[(size_t) im.ew].size());
                }
            set_size[(size_t) s] = total16 - set_off[(size_t) s];
        }
    };

    // tables that do not depend on where the images live
    const int nlanes = std::max(TC_M, (g.npack * T->per + 31) / 32 * 32);
    for (int mode = 0; mode < 2; ++mode)
    {
        g.stream = mode;
        place(mode == 1);
        const int stage = mode == 0 ? total16 : *std::max_element(set_size.begin(), set_size.end());
        g.b_stage16 = stage;
        const long long b_bytes = 16ll * (mode == 0 ? (long long) total16 * g.cgroups : 2ll * stage);
        if (b_bytes > SH_SMEM_MAX)
            continue;
        std::map<std::array<int, 3>, int> tab; // (ew, set, image width) -> first step
        std::vector<uint2> st;
        std::vector<ShGroup> groups;
        std::vector<uint32_t> rowtab((size_t) (g.nph * g.rows), 0);
        for (int ph = 0; ph < g.nph; ++ph)
            for (int i = 0; i < g.rows; ++i)
            {
                const size_t g0 = groups.size();
                for (const Range& r : all)
                {
                    if (r.phase != ph || r.i != i)
                        continue;
                    const ShImage& im = images[(size_t) r.image];
                    for (int set = 0; set < g.nsets; ++set)
                    {
                        const std::vector<ShStep>& list = steps[(size_t) r.ew][(size_t) set];
                        if (list.empty())
                            continue;
                        const int n_img = (int) im.code.size();
                        const std::array<int, 3> key = {r.ew, set, n_img};
                        auto it = tab.find(key);
                        if (it == tab.end())
                        {
                            it = tab.insert({key, (int) st.size()}).first;
                            for (const ShStep& s : list)
                            {
                                // in bounds: 128 cells from either A address, two chunks of the image
                                if (s.a1 <= s.a0 || s.a0 < 0 || s.a1 + TC_M > g.a_slot16
                                    || (s.c0 + 2) * n_img > n_img * (int) chunks[(size_t) r.ew].size())
                                    return false;
                                st.push_back(make_uint2((uint32_t) s.a0 | (uint32_t) (s.a1 - s.a0) << 16,
                                                        (uint32_t) (s.c0 * n_img) | (uint32_t) n_img << 16));
                            }
                        }
                        ShGroup gr;
                        std::memset(&gr, 0, sizeof(gr));
                        gr.dcol = (uint16_t) (set * g.set_off + r.col);
                        gr.n = (uint16_t) r.n;
                        gr.step0 = (uint16_t) it->second;
                        gr.nst = (uint16_t) list.size();
                        gr.b16 = (uint32_t) (im.off16 + r.at);
                        if (gr.dcol + gr.n > (int) TC_TMEM_COLS || r.at + r.n > n_img)
                            return false;
                        groups.push_back(gr);
                    }
                }
                rowtab[(size_t) (ph * g.rows + i)] = (uint32_t) g0 | (uint32_t) (groups.size() - g0) << 16;
            }
        if (groups.size() > 60000 || st.size() > 60000)
            return false;
        std::vector<uint2> sets;
        for (int ph = 0; ph < g.nph; ++ph)
            sets.push_back(mode == 1 ? make_uint2((uint32_t) set_off[(size_t) ph], (uint32_t) set_size[(size_t) ph])
                                     : make_uint2(0, (uint32_t) total16));
        sets.push_back(make_uint2((uint32_t) total16, 0));
        std::vector<uint32_t> items;
        const int npb = g.ipr / g.st_w;
        for (int par = 0; par < g.st_w; ++par)
            for (int pb = 0; pb < npb; ++pb)
                items.push_back((uint32_t) par | (uint32_t) (pb * 32) << 8);
        std::vector<int> lanes((size_t) nlanes, -1);
        for (int p = 0; p < g.npack * T->per; ++p)
            lanes[(size_t) p] = (p / T->per) << 16 | (p % T->per);

        auto put = [&](const void* src, size_t bytes) {
            const size_t at = T->blob.size();
            T->blob.resize(at + (bytes + 15) / 16 * 16, 0);
            std::memcpy(T->blob.data() + at, src, bytes);
            return (int) at;
        };
        T->blob.clear();
        put(st.data(), st.size() * sizeof(uint2));
        g.co_groups = put(groups.data(), groups.size() * sizeof(ShGroup)) / 16;
        g.co_rows = put(rowtab.data(), rowtab.size() * 4) / 4;
        T->too_long = T->blob.size() > (size_t) m_issue_bytes;
        if (T->too_long)
            return false; // (streamed, every image stands again and maybe others beside it: the steps are no fewer)
        T->issue.swap(T->blob);
        T->blob.clear();
        const int o_sets = put(sets.data(), sets.size() * sizeof(uint2));
        const int o_items = put(items.data(), items.size() * 4);
        const int o_lanes = put(lanes.data(), lanes.size() * 4);
        g.tab_bytes = (int) T->blob.size();
        const int bars = 8 * (2 * SH_MAX_SLOTS + 4 + 2 * g.th * g.ns) + 64;
        // staging for bulk stores (plain outputs in tiles of whole warps, at
        // most 16 filters), where three A slots still fit beside it
        const bool plain = g.e_s * g.e_r * g.e_w == 1 && g.npack == 1 && g.nb <= 16 && g.o_w % 4 == 0
                           && (g.tiles_w == 1 || g.tile_w % 32 == 0);
        int slots = 0;
        for (int stage = plain ? 1 : 0; stage >= 0 && slots == 0; --stage)
        {
            g.stage = stage ? 16 * 32 * 4 : 0;
            g.so_stage = align_up((int) b_bytes, 128);
            g.so_a = g.so_stage + SH_EPI * g.stage;
            const long long rest = SH_SMEM_MAX - 128ll - g.so_a - g.tab_bytes - bars;
            const int fit = rest < 0 ? 0 : (int) std::min<long long>(SH_MAX_SLOTS, rest / (16ll * g.a_slot16));
            g.teams = 0;
            for (int n = fit / SH_ISS * SH_ISS; n > 0; n -= SH_ISS)
            {
                int t = SH_CONV / g.ipr;
                while (n % t != 0)
                    --t;
                if (t > g.teams)
                    g.teams = t, slots = n;
            }
            // Three teams of four warps are better than two where conversion bounds: one pass of products
            // (16 -> 16 in TF32 on 100 x 100 x 75 77 / 94 us), parts of rows (16 -> 4 on 100 x 100 x 160 119 / 125), or
            // no room for two slots a team. Elsewhere they get in the way of the other roles (24 -> 24 on
            // 2 x 700 x 118 31.2 / 29.3, 16 -> 24 on 4 x 300 x 30 16.2 / 15.3, backward data 18.3 / 16.7). Over 32 forward
            // passes and 62 of backward data, 27 of them with stride 2, two teams take 0.6 and 1.2 % less (9 % at
            // best; 1.6 % more at worst, 24 -> 4 on 4 x 16 x 72 x 27).
            if (g.ipr == 4 && fit >= 6 && m_parts > 1 && (g.npack == 1 || g.tiles_w == 1))
                g.teams = 2, slots = 6;
        }
        if (slots == 0)
            continue;
        g.a_slots = slots;
        g.so_sets = g.so_a + 16 * g.a_slot16 * slots;
        g.so_items = g.so_sets + o_items - o_sets;
        g.so_lanes = g.so_sets + o_lanes - o_sets;
        g.so_bars = g.so_sets + g.tab_bytes;
        T->smem = (size_t) g.so_bars + bars + 128;
        g.nsteps = (int) st.size();
        g.ngroups = (int) groups.size();
        T->total16 = total16;
        T->packs.clear(), T->chunks.clear(), T->codes.clear();
        std::vector<int> chunk0;
        for (const auto& c : chunks)
        {
            chunk0.push_back((int) T->chunks.size());
            T->chunks.insert(T->chunks.end(), c.begin(), c.end());
        }
        for (const ShImage& im : images)
        {
            T->packs.push_back({(int) im.code.size(), (int) chunks[(size_t) im.ew].size(), chunk0[(size_t) im.ew],
                                (int) T->codes.size(), (mode == 1 ? set_off[(size_t) im.set] : 0) + im.off16});
            T->codes.insert(T->codes.end(), im.code.begin(), im.code.end());
        }
        return true;
    }
    return false;
}

// Column height, filter groups, channel groups and segments together, by the
// clocks of the busiest SM.
bool ShBuilder::build(ShTables* out) const
{
    if (!supported())
        return false;
    // (one-pass products are off by far more than their sum)
    double limit = m_parts == 1 ? SH_CHAIN_MAX : chain_limit();
    for (; limit < SH_CHAIN_MAX; limit *= 1.5)
        if (build_within(limit, out))
            return true;
    return build_within(SH_CHAIN_MAX, out);
}

// Longest chain of leading products to look for.  An fp32 FMA chain over T terms is off
// by 1.45e-8 sqrt(T), which a chain of 0.85 sqrt(T) updates on activations (they have a
// mean) and of sqrt(T) on gradients stays below.  Strided layers, and volumes with many
// channels and filters, are held to that: 16 -> 32, stride 2, 256^3, forward 3.6e-7 with
// FMAs, 6.0e-7 with 60 updates, 2.6e-7 like this (997 us against 1050); backward data 2.2e-7,
// 1.7e-6 with the corrections in the same set, 1.9e-7 like this (850 us against 960).  The
// others are not: 32 -> 32, 5 x 5, 2048 x 1024 x 2 would take 1420 us instead of 920 (1.0e-6),
// 16 -> 4 on 256^3 1050 instead of 910 (4e-7).
double ShBuilder::chain_limit() const
{
    const double terms = (double) m_cin * m_s.most() * m_r.most() * m_w.most();
    const bool strided = m_cg.stride[0] > 1 || m_cg.stride[1] > 1 || m_cg.stride[2] > 1;
    const bool as_fma = strided || (!m_flat && m_kout > 16 && m_cin >= 16);
    return as_fma ? (m_tr ? 1.0 : 0.85) * std::sqrt(terms) : SH_CHAIN_LOOSE;
}

// Few channels of a volume's dy: all three products in one chain of 45 updates (9.6e-7)
// leave twice the rows a column that two sets do (16 -> 4 on 512^3: 4420 us against 5740).
bool ShBuilder::one_set(int cgroups, int items) const
{
    return m_tr && !m_flat && m_parts == 2 && chain_limit() == SH_CHAIN_LOOSE && chain_of(3 * items, 1, cgroups) <= SH_CHAIN_LOOSE;
}

// Clocks of the busiest SM.  A fit to the times of 730 layouts of 56 passes (the layout that it
// picked of a pass was 1.7 % slower than the best of it; a maximum of products, conversion and
// draining instead of their sum: 4 %): the roles wait for one another row by row, so that
// what each of them takes adds up. The fit is older than the tables in the constant bank, blocks that both
// epilogue teams drain, and rows in parts, and has not been made again. Over passes of 40 us and more in fp32
// the time taken is 0.91 of the estimate (median; 0.62 to 1.21 for eight of ten), 0.86 where blocks are shared.
double ShBuilder::clocks(const ShGeom& g, double mma, int teams) const
{
    const double rows = (double) g.rows * g.cgroups, cells = g.cpg / m_ch * (m_kind == 0 ? 1.0 : 2.0);
    const int cell_cols = g.nb < 16 ? (g.e_s * g.e_r * g.nb + 15) / 16 : g.e_s * g.e_r * ((g.nb + 15) / 16);
    const bool bulk = g.e_s * g.e_r * g.e_w == 1 && g.npack == 1 && g.nb <= 16 && g.o_w % 4 == 0;
    const double drain = g.th * g.e_w * cell_cols * (1060.0 + (bulk ? 0.0 : 860.0)) / 2;
    double plane = 0.565 * mma + rows * (770.0 + 102.0 * cells) / teams + rows * 410.0 + drain;
    if (g.th == 1 && g.ns == (m_s.taps + m_s.st - 1) / m_s.st)
        plane += 0.63 * drain; // a block has to be drained before its plane slot is opened again
    const double waves = (double) ((g.units + m_sms - 1) / m_sms);
    // Parts of a row take more, beside whole rows, than the fit, which has none of them, says (16 -> 16 on 64^3,
    // forward with statistics: 54 us expected and 66.7 taken, 56 and 64.3 with whole rows), and more where the
    // statistics come out of the epilogue that stores them. Set by hand from a few such layers.
    const bool stats = !m_tr && !m_flat && g.kgroups == 1 && g.nb <= 16;
    const double parts = g.npack > 1 && g.tiles_w > 1 ? (stats ? 1.15 : 1.08) : 1.0;
    return parts * waves * (((g.seglen - 1) * m_s.st + m_s.taps) * plane + 16800.0);
}

// The corrections (every product but the first) are small and have a set of their own.
int ShBuilder::chain_of(int items, int lead, int cgroups) const
{
    const int steps = ((items + lead - 1) / lead + 1) / 2;
    return steps * cgroups * m_s.most() * m_r.most();
}

bool ShBuilder::build_within(double limit, ShTables* out) const
{
    std::vector<Try> tries;
    const std::vector<int> parts = row_parts();
    const int live = (m_s.taps + m_s.st - 1) / m_s.st; // planes live at once
    for (int kg = 1; kg <= 16 && kg <= m_kout; ++kg)
        for (int cgroups = 1; cgroups <= 8; cgroups *= 2)
            for (int th = m_flat ? 1 : std::min(16, m_r.q); th >= 1; --th)
            {
                ShTables T;
                Try t = {kg, th, live, cgroups, 1, 1, parts[0], 0, 0};
                if (!layout(t, &T))
                    continue;
                const int J = T.g.cpg / m_ch;
                // sets that the leading products of the cell with the most taps are dealt out to
                const int items = J * m_w.most();
                int lead = 1;
                while (lead < items && chain_of(items, lead, cgroups) > limit)
                    ++lead;
                if (chain_of(items, lead, cgroups) > limit)
                    continue;
                t.nsets = lead + (m_parts > 1 ? 1 : 0);
                if (one_set(cgroups, items))
                    t.nsets = 1;
                if (m_flat)
                {
                    // one row of blocks: spare plane slots decouple the issuer from the epilogue
                    const int cols = T.g.blk * T.g.e_w * t.nsets;
                    t.ns = std::min(16, (int) TC_TMEM_COLS / cols);
                    while (t.ns >= live
                           && align_up(t.ns * T.g.blk, 16) * T.g.e_w * t.nsets + (T.g.nb % 16 ? 16 : 0) > (int) TC_TMEM_COLS)
                        --t.ns;
                    if (t.ns < live)
                        continue;
                }
                if (!layout(t, &T))
                    continue;
                // clocks of the products of a plane's rows
                t.mma = 0;
                std::vector<std::vector<std::vector<ShStep>>> steps;
                std::vector<std::vector<ShChunk>> chunks;
                make_steps(&T, J, &steps, &chunks);
                for (int ph = 0; ph < m_s.st; ++ph)
                    for (int i = 0; i < T.g.rows; ++i)
                        for (int ew = 0; ew < T.g.e_w; ++ew)
                        {
                            size_t n = 0;
                            for (const auto& s : steps[(size_t) ew])
                                n += s.size();
                            for (const auto& r : ranges(row_code(T.g, ph, i, ew)))
                                t.mma += (double) n * sh_mma_cost(r.second) * cgroups / m_s.st;
                        }
                for (int wt : parts)
                {
                    t.wt = wt;
                    double best = 0;
                    int best_ns = 0;
                    for (int ns = 1; ns <= std::min(m_s.q, 64); ++ns)
                    {
                        Try s = t;
                        s.nseg = ns;
                        if (!layout(s, &T))
                            continue;
                        const double c = clocks(T.g, t.mma, std::max(1, SH_CONV / T.g.ipr));
                        if (best_ns == 0 || c < best)
                            best = c, best_ns = ns;
                    }
                    if (best_ns == 0)
                        continue;
                    t.nseg = best_ns;
                    t.cost = best;
                    tries.push_back(t);
                }
            }
    std::stable_sort(tries.begin(), tries.end(), [](const Try& a, const Try& b) { return a.cost < b.cost; });
    // how many converter teams fit shows in the finished tables only
    auto pick = [&](const std::vector<Try>& from) {
        int left = 24, found = 0;
        for (const Try& t : from)
        {
            if (left == 0 || found == 4 || (found > 0 && t.cost >= out->cost))
                break;
            ShTables T;
            const bool fits = layout(t, &T) && finish(t, &T);
            left -= !T.too_long; // (lower columns have shorter tables)
            if (fits)
            {
                // two teams of four are taken where three would be slower (finish), which the fit does not know:
                // priced as the three that it would have liked better
                T.cost = clocks(T.g, t.mma, T.g.ipr == 4 && T.g.teams == 2 ? 3 : T.g.teams);
                T.chain = T.g.nsets == 1 ? chain_of(m_parts * (m_parts + 1) / 2 * T.g.cpg / m_ch * m_w.most(), 1, T.g.cgroups)
                                         : chain_of(T.g.cpg / m_ch * m_w.most(), T.g.nsets - (m_parts > 1 ? 1 : 0), T.g.cgroups);
                if (found++ == 0 || T.cost < out->cost)
                    *out = T;
            }
        }
        return found > 0;
    };
    std::vector<Try> whole;
    for (const Try& t : tries)
        if (t.wt == parts[0])
            whole.push_back(t);
    const bool found = pick(whole);
    if (whole.size() == tries.size() || !found)
        return found;
    const ShTables rows = *out;
    if (!pick(tries) || out->cost > rows.cost)
        *out = rows;
    // The CUDA-core kernels are weighed against whole rows, which their rule was made with. (Layers in parts
    // take 0.63 of that, so that a layer near the line may be on the CUDA cores that would be faster here.)
    out->cost = rows.cost;
    return true;
}

} // namespace dcb
