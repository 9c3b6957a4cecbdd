// tcgen05 backward filter (strides 1 or 2 per dimension, dilation 1):
//
//   dw[k][c][kd][kh][kw] = sum over (n, od, oh, ow) dy[n][k][od][oh][ow] *
//                          x[n][c][od*sd+kd-pd][oh*sh+kh-ph][ow*sw+kw-pw]
//
// GEMM view: the reduction runs along W, eight positions per instruction, both
// operands K-major in shared memory without swizzle (a cell is 16 bytes = four
// positions of one row).
//   A  rows (x row, part, kw, c): an input row once per tap kw, shifted by it, so
//      that no address has to move by less than a cell
//   B  rows (dy row, part, k)
// `part` is the hi or the lo half of a two-way TF32 split.  One instruction
// multiplies `A` consecutive input rows (up to 128 matrix rows) with `nb`
// consecutive dy rows, all pairs at once; pair (a, b) is tap kh = a - b * sh, pairs
// that are no tap are not read.  Rows of both operands are plentiful this way (4
// channels x 3 taps x 2 parts x 5 input rows = 120 of 128, 3 dy rows x 16 filters x
// 2 parts = 96 columns), where a plain im2col product of a layer with few channels
// and filters would use a fraction of both.
//
// A stage is B dy rows and the X = (B - 1) * sh + fh input rows of each of its kd
// planes, PW positions wide, in one of two to eight shared-memory buffers.
// Few channels leave room for the accumulators of all kd in one role.  The stages then
// walk along D (`ring`): a stage brings one plane of x and its dy rows, the kd planes are
// those of the last kdg stages, and an input row is read, split and written once instead
// of once per kd; the first kdg - 1 steps of a walk only bring x.
// Converter warps read x and dy straight from global memory, split them and write
// the stage; one thread issues.  What does not fit tensor memory (512 columns,
// accumulators and running sums) or the 128 matrix rows is dealt out in roles:
// groups of channels, planes kd or filters, a CTA always working for one, and
// launches for groups of taps kw.
//
// The tensor pipe adds into its fp32 accumulators by truncation: after
// WG_CHAIN updates four warps add the hi columns into running sums beside them,
// rounding to nearest, and zero them (the lo columns are 2^-11 of the result: their
// chains may run to the end).
// At the end every CTA reduces its accumulators to its part of the filter and
// wg_fold_kernel adds the CTAs' parts in order, in fp64: the same result every run.
#pragma once

#include "conv_tc_wgrad_api.cuh"

namespace dcb
{

struct WgUnit
{
    int n, od, h0, w0;
};

template <bool RING>
__device__ __forceinline__ WgUnit wg_unit(const WgGeom& g, long long s)
{
    WgUnit u;
    uint32_t r = (uint32_t) s;
    if (RING)
    {
        u.od = (int) (r % (uint32_t) g.out[0]);
        r /= (uint32_t) g.out[0];
    }
    u.h0 = (int) (r % (uint32_t) g.hblocks) * g.B;
    r /= (uint32_t) g.hblocks;
    u.w0 = (int) (r % (uint32_t) g.wchunks) * g.PW;
    r /= (uint32_t) g.wchunks;
    if (!RING)
    {
        u.od = (int) (r % (uint32_t) g.out[0]);
        r /= (uint32_t) g.out[0];
    }
    u.n = (int) r;
    return u;
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

// The registers of two tensor-memory loads may be read after this.
__device__ __forceinline__ void tmem_loaded(uint32_t (&a)[8], uint32_t (&b)[8])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                   "+r"(b[0]), "+r"(b[1]), "+r"(b[2]), "+r"(b[3]), "+r"(b[4]), "+r"(b[5]), "+r"(b[6]), "+r"(b[7])
                 :
                 : "memory");
}

__device__ __forceinline__ void st_v4(uint32_t dst, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

struct WgConvArgs
{
    uint32_t base, full_s, empty_s;
    const uint4* itab;
    int items, warps, rc, rkw, rkd, rk, s0, s1, w, lane;
    volatile int* abort_flag;
};

// Converters.  Some warps read x, the others dy; warp w of `warps` takes two items at
// a time (w, w + warps; then the next two), loads one pair ahead.  A lane is four
// positions of one channel or filter; the cells behind them are fetched as the aligned
// 16-byte pieces they lie in, the first one AL cells below them (AL < 0: cell by cell).
// Lanes outside the tensor store zeros (the padding).  Eight lanes along a row, then the
// next channel: a quarter of a 16-byte load is then one line of 128 bytes, and a quarter of
// a store is eight cells LBO = 16 mod 128 apart.  (With the channels side by side a quarter
// touched the same banks of four lines: 256^3, 4 -> 16 1206 -> 1011 us, 128^3 185 -> 148,
// 32 -> 32 on 24 x 40 x 64 119 -> 111.)  A warp's own chain of dependent
// instructions is what bounds a stage where channels are few: hence pairs of items
// without branches between them, and stages that follow each other along H, so that
// most of them only move a pointer.
template <bool ISX, int SW, int KWG, int AL, bool RING>
__device__ __forceinline__ bool wg_convert(const WgGeom& g, const WgConvArgs& c, const float* __restrict__ src)
{
    constexpr int NV = ISX ? 3 * SW + KWG : 4;                  // cells behind four positions
    constexpr int AO = AL < 0 ? 0 : AL, NB = (NV + AO + 3) / 4; // their offset in the pieces, pieces
    constexpr uint32_t ALL = (1u << NV) - 1;
    const int cl = c.lane >> 3, ql = c.lane & 7;
    const uint32_t lane_dst = (uint32_t) (ql * (ISX ? g.lbo_x : g.lbo_y) + 16 * cl);
    const uint32_t row16 = 16u * (uint32_t) (ISX ? g.cg : g.kgp);
    const int rows_in = ISX ? g.in[1] : g.out[1], step_rows = ISX ? g.B * g.stride[1] : g.B;
    const long long step = RING ? 4ll * (ISX ? g.xs[0] : g.ys[0]) : 4ll * step_rows * (ISX ? g.xs[1] : g.ys[1]);
    int seg = 0, seg_left = 0, odv = 0; // RING: stages and steps of a walk along D, dy plane of the step in it
    // Pairs in flight.  dy of a walk along D comes from as many distant places as there are
    // filters and takes few registers: four (256^3, 4 -> 16 channels: 1284 -> 1179 us); along
    // H the next rows are near and more only costs (stride 2: 1084 -> 1108 us).
    constexpr int AHEAD = !ISX && RING ? 4 : 2;
    float t[AHEAD][2][4 * NB];
    uint32_t dst[AHEAD][2] = {}, mask[AHEAD][2] = {};
    uint32_t wait[AHEAD] = {}, tell[AHEAD] = {};
    bool has[AHEAD] = {};
    int item = c.w - 2 * c.warps, s = c.s0, buf = 0;
    uint32_t lap = 0, st = c.base;
    bool ok = true, more = c.s0 < c.s1, fresh = true;
    const char* b0 = nullptr; // the stage's first cells, this lane's channel and positions
    int h0 = 0, r0 = 0, id0 = 0;
    uint32_t m8[2] = {0, 0}; // valid cells, per group of eight lanes along the row
    auto locate = [&]() {
        WgUnit u = wg_unit<RING>(g, s);
        if (RING)
        {
            seg = min(c.s1 - s, g.out[0] - u.od);
            seg_left = seg + g.kdg - 1;
            odv = 1 - g.kdg;
            if (!ISX)
                u.od += odv;
        }
        h0 = u.h0;
        const int w0 = ISX ? u.w0 * SW + c.rkw - g.pad[2] : u.w0, width = ISX ? g.in[2] : g.out[2];
        if (ISX)
        {
            id0 = u.od * g.stride[0] + c.rkd - g.pad[0];
            r0 = u.h0 * g.stride[1] - g.pad[1];
            b0 = reinterpret_cast<const char*>(src + (long long) u.n * g.xs_n + (long long) (c.rc + cl) * g.xs_c
                                               + (long long) id0 * g.xs[0] + (long long) r0 * g.xs[1] + w0 + 4 * ql * SW - AO);
        }
        else
        {
            r0 = u.h0;
            b0 = reinterpret_cast<const char*>(src + (long long) u.n * g.ys_n + (long long) (c.rk + cl) * g.ys_c
                                               + (long long) u.od * g.ys[0] + (long long) r0 * g.ys[1] + w0 + 4 * ql);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
        {
            const int iw = w0 + (4 * ql + 32 * i) * (ISX ? SW : 1);
            uint32_t m = ALL;
            if (iw < 0)
                m = iw <= -NV ? 0u : m << -iw & m;
            if (iw + NV > width)
                m = iw >= width ? 0u : m & ((1u << (width - iw)) - 1);
            m8[i] = ql + 8 * i < g.Q ? m : 0u;
        }
    };
    if (more)
        locate();
#pragma unroll 1
    while (ok && (more || has[0]))
    {
#pragma unroll
        for (int q = 0; q < AHEAD; ++q)
        {
            if (has[q])
            {
                if (wait[q] != 0)
                    ok = ok && mbar_wait_s<20>(wait[q] & ~7u, wait[q] & 1u, c.abort_flag);
                // tensor edges: cells that do not exist (and were not loaded) are zeros
                if (__any_sync(0xffffffffu, mask[q][0] != ALL || mask[q][1] != ALL))
                {
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int e = 0; e < NV; ++e)
                            t[q][i][AO + e] = mask[q][i] >> e & 1 ? t[q][i][AO + e] : 0.f;
                }
#pragma unroll
                for (int i = 0; i < 2; ++i)
                {
                    uint32_t hi[NV], lo[NV];
#pragma unroll
                    for (int e = 0; e < NV; ++e)
                    {
                        hi[e] = tf32_rna(t[q][i][AO + e]);
                        // exact remainder below 2^-11 |x|; the pipe reads its upper 19 bits
                        lo[e] = __float_as_uint(t[q][i][AO + e] - __uint_as_float(hi[e]));
                    }
                    if (dst[q][i] != 0 && ok)
                    {
                        uint32_t d = dst[q][i];
                        if (ISX)
                        {
#pragma unroll
                            for (int kw = 0; kw < KWG; ++kw, d += row16)
                                st_v4(d, hi[kw], hi[kw + SW], hi[kw + 2 * SW], hi[kw + 3 * SW]);
#pragma unroll
                            for (int kw = 0; kw < KWG; ++kw, d += row16)
                                st_v4(d, lo[kw], lo[kw + SW], lo[kw + 2 * SW], lo[kw + 3 * SW]);
                        }
                        else
                        {
                            st_v4(d, hi[0], hi[1], hi[2], hi[3]);
                            st_v4(d + row16, lo[0], lo[1], lo[2], lo[3]);
                        }
                    }
                }
                if (tell[q] != 0)
                {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (c.lane == 0)
                        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tell[q]) : "memory");
                }
                has[q] = false;
            }
            if (!more)
                continue;
            wait[q] = 0;
            item += 2 * c.warps;
            if (item >= c.items || fresh)
            {
                if (!fresh)
                {
                    item = c.w;
                    if (RING)
                        s += --seg_left == 0 ? seg : 0;
                    else
                        ++s;
                    if (s == c.s1)
                    {
                        more = false;
                        continue;
                    }
                    st += (uint32_t) g.stage_bytes;
                    if (++buf == g.nstages)
                    {
                        buf = 0;
                        st = c.base;
                        ++lap;
                    }
                    h0 += g.B;
                    if (RING && seg_left != 0)
                    {
                        // the next plane
                        ++id0;
                        ++odv;
                        b0 += step;
                    }
                    else if (!RING && h0 < g.out[1])
                    {
                        // the next rows of the same column
                        r0 += step_rows;
                        b0 += step;
                    }
                    else
                        locate();
                }
                fresh = false;
                if (lap > 0)
                    wait[q] = (c.empty_s + 8u * (uint32_t) buf) | ((lap - 1) & 1u);
            }
            tell[q] = item + 2 * c.warps >= c.items ? c.full_s + 8u * (uint32_t) buf : 0u;
            has[q] = true;
            uint4 it[2];
            it[0] = c.itab[item];
            it[1] = item + c.warps < c.items ? c.itab[item + c.warps] : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int i = 0; i < 2; ++i)
            {
                const int row = (int) (it[i].x >> 8 & 255u);
                const bool second = (it[i].x >> 24) != 0; // group of lanes along the row
                const bool stored = cl < (int) (it[i].x >> 16 & 15u) && (second ? ql + 8 : ql) < g.Q;
                bool in = cl < (int) (it[i].x >> 20 & 15u) && (unsigned) (r0 + row) < (unsigned) rows_in;
                if (RING && !ISX)
                    in = in && odv >= 0;
                if (ISX)
                    in = in && (unsigned) (id0 + (int) (it[i].x >> 2 & 63u)) < (unsigned) g.in[0];
                const uint32_t m = in ? (second ? m8[1] : m8[0]) : 0u;
                dst[q][i] = stored ? st + it[i].y + lane_dst : 0u;
                mask[q][i] = m;
                const float* p = reinterpret_cast<const float*>(b0) + it[i].z;
                if (AL >= 0)
                {
#pragma unroll
                    for (int e = 0; e < NB; ++e)
                    {
                        // the valid cells among the piece's
                        const int first = 4 * e - AO;
                        const uint32_t bits = first >= 0 ? m >> (first >= 0 ? first : 0) & 15u
                                                         : m & (15u >> (first < 0 ? -first : 0));
                        if (bits != 0)
                        {
                            const float4 f = __ldg(reinterpret_cast<const float4*>(p) + e);
                            t[q][i][4 * e] = f.x, t[q][i][4 * e + 1] = f.y, t[q][i][4 * e + 2] = f.z,
                                           t[q][i][4 * e + 3] = f.w;
                        }
                    }
                }
                else
                {
#pragma unroll
                    for (int e = 0; e < NV; ++e)
                        if (m >> e & 1)
                            t[q][i][e] = __ldg(p + e);
                }
            }
        }
    }
    return ok;
}

// One launch per group of taps kw (rkw is the first): where a lane's cells start
// inside a 16-byte piece is then the same for all, and the converters are compiled
// for it.
template <int SW, int KWG, int AL>
__global__ void __launch_bounds__(WG_THREADS, 1)
    wg_conv_kernel(const __grid_constant__ WgGeom g, const float* __restrict__ x, const float* __restrict__ dy,
                   float* __restrict__ part, int* status, int rkw)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + g.so_bars); // [nstages] converters -> issuer
    uint64_t* empty = full + WG_MAX_STAGES;                         // [nstages] issuer -> converters
    uint64_t* chain_end = empty + WG_MAX_STAGES;                    // issuer -> running sums
    uint64_t* cleared = chain_end + 1;                              // running sums -> issuer
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(cleared + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int items = g.items_x + g.items_y;
    const int role = (int) blockIdx.x % g.roles, slice = (int) blockIdx.x / g.roles;
    const int rc = role % g.ncg * g.cg, rkd = role / g.ncg % g.nkd * g.kdg, rk = role / (g.ncg * g.nkd) * g.kg;
    const int s0 = (int) (g.stages * slice / g.parts), s1 = (int) (g.stages * (slice + 1) / g.parts);

    if (tid == 0)
    {
        for (int s = 0; s < WG_MAX_STAGES; ++s)
        {
            mbar_init(&full[s], (uint32_t) (min(g.items_x, g.warps_x) + min(g.items_y, WG_CONV - g.warps_x)));
            mbar_init(&empty[s], 1);
        }
        mbar_init(chain_end, 1);
        mbar_init(cleared, WG_FLUSH);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0)
    {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(TC_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    WgTile* tiles = reinterpret_cast<WgTile*>(smem + g.so_tiles);
    for (int i = tid; i < g.ntiles; i += WG_THREADS)
        tiles[i] = g.tiles[i];
    // warp items of a stage: what and how many channels or filters, where it goes, where it comes from
    uint4* itab = reinterpret_cast<uint4*>(smem + g.so_items);
    for (int i = tid; i < items; i += WG_THREADS)
    {
        const bool isx = i < g.items_x;
        int r = isx ? i : i - g.items_x;
        const int q0 = r % g.qg * 8;
        r /= g.qg;
        const int ch = r % (isx ? g.cq : g.kq) * 4;
        r /= isx ? g.cq : g.kq; // kd * X + a, or b
        const int kd = isx ? r / g.X : 0, row = isx ? r - kd * g.X : r;
        // rows of the operand that exist (the others hold zeros), and of those the ones the tensor has
        const int rows = min(4, (isx ? g.cg : g.kg) - ch);
        const int real = max(0, min(rows, isx ? g.c - rc - ch : g.k - rk - ch));
        const long long off = isx ? ch * g.xs_c + kd * g.xs[0] + row * g.xs[1] + 4 * q0 * SW
                                  : ch * g.ys_c + row * g.ys[1] + 4 * q0;
        itab[i] = make_uint4((isx ? 1u : 2u) | (uint32_t) kd << 2 | (uint32_t) row << 8 | (uint32_t) rows << 16
                                 | (uint32_t) real << 20 | (uint32_t) q0 << 24,
                             (uint32_t) (isx ? q0 * g.lbo_x + 16 * (r * g.r8 + ch)
                                             : g.y_off + q0 * g.lbo_y + 16 * (r * g.n8 + ch)),
                             (uint32_t) off, 0u); // (elements, below 2^32: wg_layout)
    }
    // Matrix rows that no item writes (filters up to a multiple of 8, rows past a tile's) hold what an
    // earlier kernel left: they only reach accumulators that nobody reads.
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // accumulators, running sums (all 512 columns in a loop that is not unrolled: two registers fewer spilled with
    // three taps, large layers the same, small ones 10 % slower)
    const uint32_t columns = (uint32_t) (g.sum_col + g.kdg * g.nblocks * g.kgp);
    if (warp < 4)
        for (uint32_t c = 0; c < columns; c += 16)
            tmem_st16_zero(tmem + ((uint32_t) (warp * 32) << 16) + c);
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    bool ok = true;

    if (warp < WG_FLUSH)
    {
        // running sums, pieces of eight hi columns
        const uint32_t la = tmem + ((uint32_t) ((warp & 3) * 32) << 16);
        const int pieces = g.kgp / 8, total = g.kdg * g.nblocks * pieces;
        uint32_t par = 0;
        for (int s = s0 + g.flush_stages; s < s1 && ok; s += g.flush_stages, par ^= 1)
        {
            ok = mbar_wait_t<500>(chain_end, par, abort_flag);
            if (!ok)
                break;
            tc_fence_after();
            // two pieces at a time: a load takes some hundred clocks whatever it brings
#pragma unroll 1
            for (int i = 0; i < total; i += 2)
            {
                uint32_t d[2], r[2], a[2][8], b[2][8];
#pragma unroll
                for (int h = 0; h < 2; ++h)
                {
                    const int k = min(i + h, total - 1), block = k / pieces, p8 = (k - block * pieces) * 8;
                    d[h] = la + (uint32_t) (block / g.nblocks * g.kd_cols + block % g.nblocks * g.n8 + p8);
                    r[h] = la + (uint32_t) (g.sum_col + block * g.kgp + p8);
                    tmem_ld8(d[h], a[h]);
                    tmem_ld8(r[h], b[h]);
                }
                tmem_loaded(a[0], b[0]);
                tmem_loaded(a[1], b[1]);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                {
                    uint32_t v[8], z[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        v[j] = __float_as_uint(__uint_as_float(a[h][j]) + __uint_as_float(b[h][j])), z[j] = 0u;
                    if (i + h < total)
                    {
                        tmem_st8(r[h], v);
                        tmem_st8(d[h], z);
                    }
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(cleared);
        }
    }
    else if (warp < WG_ISSUE_WARP)
    {
        const int w = warp - WG_FLUSH;
        const bool isx = w < g.warps_x;
        const WgConvArgs c = {smem_u32(smem), smem_u32(full), smem_u32(empty), isx ? itab : itab + g.items_x,
                              isx ? g.items_x : g.items_y, isx ? g.warps_x : WG_CONV - g.warps_x, rc, rkw, rkd, rk, s0, s1,
                              isx ? w : w - g.warps_x, lane, abort_flag};
        if (c.w < c.items)
        {
            if (g.ring)
            {
                if (!isx)
                    ok = g.vec_y ? wg_convert<false, 1, 1, 0, true>(g, c, dy) : wg_convert<false, 1, 1, -1, true>(g, c, dy);
                else
                    ok = wg_convert<true, SW, KWG, AL, true>(g, c, x);
            }
            else if (!isx)
                ok = g.vec_y ? wg_convert<false, 1, 1, 0, false>(g, c, dy) : wg_convert<false, 1, 1, -1, false>(g, c, dy);
            else
                ok = wg_convert<true, SW, KWG, AL, false>(g, c, x);
        }
    }
    else
    {
        // issuer
        uint32_t elected;
        asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(elected));
        const uint32_t base16 = smem_u32(smem) >> 4, dhi = 8u | (1u << 14); // SBO 128 bytes, descriptor version
        const uint32_t lx = (uint32_t) g.lbo_x >> 4, ly = (uint32_t) g.lbo_y >> 4;
        const int ksteps = g.Q / 2;
        int buf = 0, left = g.flush_stages;
        uint32_t par = 0, cpar = 0;
        // ring: `lead` steps of a walk only bring planes of x; a step's buffer is free again when the
        // last step that reads its plane is through
        const int lead = g.ring ? g.kdg - 1 : 0;
        int walk = lead, walk_end = 0, steps = 0; // position in the walk, its length
#pragma unroll 1
        for (int s = s0; s < s1 && ok;)
        {
            if (g.ring && walk_end == 0)
                walk = 0, walk_end = min(s1 - s, g.out[0] - s % g.out[0]) + lead;
            const bool real = walk >= lead;
            if (real && left == 0)
            {
                if (elected)
                    mma_commit(chain_end);
                ok = mbar_wait_t<0>(cleared, cpar, abort_flag);
                cpar ^= 1;
                left = g.flush_stages;
                if (!ok)
                    break;
            }
            left -= real;
            ok = mbar_wait_t<0>(&full[buf], par, abort_flag);
            if (!ok)
                break;
            tc_fence_after();
            const uint32_t b_st = base16 + (uint32_t) (buf * g.stage_bytes + g.y_off) / 16u;
            const int oldest = buf - lead + (buf < lead ? g.nstages : 0);
            if (elected)
            {
                int xb = oldest;
#pragma unroll 1
                for (int kd = 0; kd < g.kdg && real; ++kd)
                {
                    const uint32_t a_st =
                        base16 + (uint32_t) (xb * g.stage_bytes) / 16u + (g.ring ? 0u : (uint32_t) (kd * g.kd_a16));
                    if (g.ring && ++xb == g.nstages)
                        xb = 0;
#pragma unroll 1
                    for (int t = 0; t < g.ntiles; ++t)
                    {
                        const WgTile tl = tiles[t];
                        uint32_t a = (a_st + tl.a16) | lx << 16;
                        uint32_t b = (b_st + tl.b16) | ly << 16;
                        const uint32_t d = tmem + tl.dcol + (uint32_t) (kd * g.kd_cols);
#pragma unroll 4
                        for (int ks = 0; ks < ksteps; ++ks)
                        {
                            asm volatile("{\n\t.reg .pred t;\n\tsetp.eq.b32 t, 0, 0;\n\t"
                                         "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, t;\n\t}" ::"r"(d),
                                         "l"((uint64_t) dhi << 32 | a), "l"((uint64_t) dhi << 32 | b), "r"(tl.idesc));
                            a += 2 * lx;
                            b += 2 * ly;
                        }
                    }
                }
                if (steps >= lead)
                    mma_commit(&empty[oldest]);
                if (real && s + 1 == s1)
                    mma_commit(chain_end);
            }
            __syncwarp();
            ++steps;
            s += real;
            if (g.ring && ++walk == walk_end)
                walk_end = 0;
            if (++buf == g.nstages)
            {
                buf = 0;
                par ^= 1;
            }
        }
    }

    // every role has left its loop (all waits are bounded and watch the abort
    // flag); the last instructions' completion is one more phase of chain_end
    __syncthreads();
    if (ok && s1 > s0)
        ok = mbar_wait(chain_end, (uint32_t) ((s1 - s0 - 1) / g.flush_stages) & 1, abort_flag);
    tc_fence_after();
    // reduction, one kd plane at a time: accumulators to shared memory (the
    // stages' space) as [column][lane], then every output adds its pairs
    float* dump = reinterpret_cast<float*>(smem);
    const int fh = g.f[1], per_kd = g.kg * g.cg * fh * KWG;
    float* out = part + (long long) blockIdx.x * g.kdg * per_kd;
#pragma unroll 1
    for (int kd = 0; kd < g.kdg; ++kd)
    {
        if (warp < WG_FLUSH)
        {
            const uint32_t la = tmem + ((uint32_t) ((warp & 3) * 32) << 16);
            const int l = (warp & 3) * 32 + lane;
#pragma unroll 1
            for (int c8 = 0; c8 < g.nblocks * g.n8; c8 += 8)
            {
                uint32_t a[8], b[8];
                tmem_ld8(la + (uint32_t) (kd * g.kd_cols + c8), a);
                const int block = c8 / g.n8, in = c8 - block * g.n8;
                if (in < g.kgp)
                    tmem_ld8(la + (uint32_t) (g.sum_col + (kd * g.nblocks + block) * g.kgp + in), b);
                else
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        b[j] = 0u;
                tmem_loaded(a, b);
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    dump[(c8 + j) * 128 + l] = __uint_as_float(a[j]) + __uint_as_float(b[j]);
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int e = tid; e < per_kd; e += WG_THREADS)
        {
            // lanes of a warp walk (kw, c): neighbouring columns of shared memory
            const int c = e % g.cg, kw = e / g.cg % KWG, kh = e / (g.cg * KWG) % fh, k = e / (g.cg * KWG * fh);
            double sum = 0.0;
#pragma unroll 1
            for (int r = 0; r < g.nclasses; ++r)
#pragma unroll 1
                for (int al = 0; al < g.A; ++al)
                {
                    const int num = r + al - kh;
                    int delta = num;
                    if (g.stride[1] == 2)
                    {
                        if (num & 1)
                            continue;
                        delta = num >> 1;
                    }
                    const int i = delta - g.class_lo[r];
                    if (i < 0 || i >= g.class_n[r])
                        continue;
                    const float* col = dump + (g.class_col[r] + i * g.n8 + k) * 128 + al * g.r8 + kw * g.cg + c;
                    const int lo_k = g.kgp * 128, lo_x = KWG * g.cg;
                    sum += (double) col[0] + ((double) col[lo_x] + (double) col[lo_k]) + (double) col[lo_k + lo_x];
                }
            out[(((long long) k * g.cg + c) * g.kdg + kd) * fh * KWG + kh * KWG + kw] = (float) sum;
        }
        __syncthreads();
    }
    if (!ok && lane == 0)
        atomicExch(status, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_TMEM_COLS) : "memory");
}

template <int SW, int KWG, int AL>
int32_t wg_launch(const WgGeom& g, int rkw, const float* x, const float* dy, float* part, int* status, cudaStream_t stream)
{
    auto kernel = wg_conv_kernel<SW, KWG, AL>;
    const size_t smem = g.smem < 120 * 1024 ? 120 * 1024 : (size_t) g.smem; // one CTA per SM: it owns all of tensor memory
    const int32_t set = allow_dynamic_smem(reinterpret_cast<const void*>(kernel), 227 * 1024);
    if (set != DCB_OK)
        return set;
    kernel<<<(unsigned) (g.roles * g.parts), WG_THREADS, smem, stream>>>(g, x, dy, part, status, rkw);
    DCB_LAUNCH_CHECK();
    return DCB_OK;
}

template <int SW, int KWG>
int32_t wg_launch_at(const WgGeom& g, int al, int rkw, const float* x, const float* dy, float* part, int* status,
                     cudaStream_t stream)
{
    switch (al)
    {
    case 0: return wg_launch<SW, KWG, 0>(g, rkw, x, dy, part, status, stream);
    case 1: return wg_launch<SW, KWG, 1>(g, rkw, x, dy, part, status, stream);
    case 2: return wg_launch<SW, KWG, 2>(g, rkw, x, dy, part, status, stream);
    case 3: return wg_launch<SW, KWG, 3>(g, rkw, x, dy, part, status, stream);
    default: return wg_launch<SW, KWG, -1>(g, rkw, x, dy, part, status, stream);
    }
}

} // namespace dcb
