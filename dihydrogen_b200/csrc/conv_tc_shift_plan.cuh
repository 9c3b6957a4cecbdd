// Host side of the shift kernel: from a convolution's geometry to its tables
// (see conv_tc_shift.cuh for what the kernel does with them).
#pragma once

#include "conv_simt.cuh"
#include "conv_tc_shift.cuh"

#include <algorithm>
#include <array>
#include <cmath>
#include <map>
#include <vector>

namespace dcb
{

// One k-step: two 16-byte cells of the A slot and two of the filter image.
struct ShChunk // one cell of the filter image: 4 or 8 channels of one tap
{
    int part, kw, ch; // part < 0: zeros
    bool operator==(const ShChunk& o) const { return part == o.part && kw == o.kw && ch == o.ch; }
};

struct ShStep
{
    int a0, a1; // 16-byte units in the A slot, a1 > a0
    int c0;     // chunk pair c0, c0 + 1
};

struct ShImage
{
    int ew;
    std::vector<int> code; // per column: filter << 16 | tap base, or -1
    int set;               // phase (streamed) or 0
    int off16;             // in its set
};

struct ShAxis // taps of one dimension in staged terms
{
    int in, q, o, st, e, taps, pad;
    // filter tap that staged tap t contributes to cell e, or -1
    int k(int t, int e_) const { return map[(size_t) e_ * taps + t]; }
    // taps of the cell that has the most
    int most() const
    {
        int m = 0;
        for (int c = 0; c < e; ++c)
            m = std::max(m, (int) std::count_if(map.begin() + c * taps, map.begin() + (c + 1) * taps, [](int v) { return v >= 0; }));
        return m;
    }
    std::vector<int> map;
};

struct ShPack // filter-image kernel's tables
{
    int n, nchunks, chunk0, code0, off16;
};

struct ShTables
{
    ShGeom g;
    int per;                         // positions staged for a sub-column
    int kind, parts;
    bool wide;                       // 64-bit channel offsets
    int c_of_cell;
    size_t smem;
    double cost;                     // of the best layout without parts of rows
    int chain;                       // longest chain of leading products in one accumulator
    std::vector<uint8_t> issue;      // issuers' tables
    bool too_long = false;           // they would not fit
    std::vector<uint8_t> blob;       // the other roles' tables, which the kernel copies to shared memory
    std::vector<ShPack> packs;       // filter images
    std::vector<ShChunk> chunks;
    std::vector<int> codes;
    int total16;                     // 16-byte units of one (filter group, channel group)
    ShExact exact;                   // without the tensors and alpha
    long long w_ko, w_ci;            // strides of the filter tensor
};

inline int floor_div(int a, int b)
{
    return a >= 0 ? a / b : -((-a + b - 1) / b);
}

inline ShAxis sh_axis(int in, int out, int f, int stride, int pad, bool transposed)
{
    ShAxis x;
    if (!transposed)
    {
        x.in = in, x.q = x.o = out, x.st = stride, x.e = 1, x.taps = f, x.pad = pad;
        for (int t = 0; t < f; ++t)
            x.map.push_back(t);
        return x;
    }
    // dx[s * a + e] takes dy[o] through tap k = s * a + e + pad - s * o: with
    // o = a + lo + t, k = e + pad - s * (lo + t)
    const int lo = -floor_div(f - 1 - pad, stride), hi = floor_div(stride - 1 + pad, stride);
    x.in = out, x.o = in, x.q = (in + stride - 1) / stride, x.st = 1, x.e = stride, x.taps = hi - lo + 1, x.pad = -lo;
    for (int e = 0; e < stride; ++e)
        for (int t = 0; t < x.taps; ++t)
        {
            const int k = e + pad - stride * (lo + t);
            x.map.push_back(k >= 0 && k < f ? k : -1);
        }
    return x;
}

// clocks of one instruction of width n (measured, shared-memory operands)
inline double sh_mma_cost(int n)
{
    return std::max(45.5, std::max(n / 2.0, 32.0 + n / 4.0));
}

class ShBuilder
{
public:
    // issue_bytes: what the issuers' tables may take, SH_CONST at most
    ShBuilder(const ConvGeom& cg, bool transposed, int math_mode, int sms, int issue_bytes = SH_CONST)
        : m_cg(cg), m_tr(transposed), m_sms(sms), m_issue_bytes(std::min(issue_bytes, (int) SH_CONST))
    {
        m_flat = cg.in[0] == 1 && cg.out[0] == 1 && cg.f[0] == 1 && cg.pad[0] == 0 && cg.stride[0] == 1;
        const int s = m_flat ? 1 : 0;
        m_s = axis(s);
        m_r = m_flat ? sh_axis(1, 1, 1, 1, 0, false) : axis(1);
        m_w = axis(2);
        m_cin = transposed ? cg.k : cg.c;
        m_kout = transposed ? cg.c : cg.k;
        m_fp32 = math_mode == DCB_MATH_FP32;
        m_bf16 = math_mode == DCB_MATH_BF16;
        // cells of four channels keep narrow inputs from padding half a cell
        m_kind = (m_cin <= 4 || math_mode == DCB_MATH_TF32) ? 0 : 1;
        m_parts = !m_fp32 ? 1 : (m_kind == 0 ? 2 : 3);
        m_ch = m_kind == 0 ? 4 : 8;
    }

    bool supported() const
    {
        for (int i = 0; i < 3; ++i)
            if (m_cg.dil[i] != 1 || m_cg.stride[i] < 1 || m_cg.stride[i] > 2 || m_cg.pad[i] > m_cg.f[i] - 1
                || m_cg.f[i] > 16)
                return false;
        return (long long) m_cg.n * m_cg.out[0] * m_cg.out[1] * m_cg.out[2] > 0
               && (long long) m_cg.n * m_cg.in[0] * m_cg.in[1] * m_cg.in[2] > 0 && m_cin > 0 && m_kout > 0
               && m_w.taps <= 24;
    }

    bool build(ShTables* out) const;

private:
    ShAxis axis(int i) const
    {
        return sh_axis(m_cg.in[i], m_cg.out[i], m_cg.f[i], m_cg.stride[i], m_cg.pad[i], m_tr);
    }
    struct Try
    {
        int kg, th, ns, cgroups, nsets, nseg, wt;
        double cost, mma;
    };
    double chain_limit() const;
    double clocks(const ShGeom& g, double mma, int teams) const;
    bool one_set(int cgroups, int items) const;
    int packed(int w) const;
    std::vector<int> row_parts() const;
    int chain_of(int items, int lead, int cgroups) const;
    bool build_within(double limit, ShTables* out) const;
    bool layout(const Try& t, ShTables* T) const;
    void make_steps(ShTables* T, int J, std::vector<std::vector<std::vector<ShStep>>>* steps,
                    std::vector<std::vector<ShChunk>>* chunks) const;
    std::vector<std::pair<int, int>> ranges(const std::vector<int>& code) const;
    std::vector<int> row_code(const ShGeom& g, int phase, int i, int ew) const;
    bool finish(const Try& t, ShTables* T) const;

    ConvGeom m_cg;
    bool m_tr, m_flat, m_fp32, m_bf16;
    int m_sms, m_issue_bytes, m_cin, m_kout, m_kind, m_parts, m_ch;
    ShAxis m_s, m_r, m_w;
};

} // namespace dcb
