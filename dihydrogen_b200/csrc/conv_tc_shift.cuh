// tcgen05 convolution whose A operand lives in shared memory pixel by pixel
// ("shift kernel"): forward and backward data, strides 1 and 2.
//
// A staged input row is written once, as planes of 16-byte cells: cell = one
// position along W, 4 (TF32) or 8 (bf16) channels of one part of the split
// operand.  Consecutive positions are consecutive cells, which is the K-major
// layout without swizzle (rows of a core matrix 16 bytes apart, SBO = 128), so
// tap kw of the same row is the same operand with its start address moved by kw
// cells: nothing is re-materialised per tap.  A k-step is two such cells (LBO =
// the distance between them), whatever two planes or shifts they come from.
//
// Precision of the products: one pass on TF32 or bf16 operands, or fp32 quality
// as 3 products of a two-way TF32 split (few channels) or 6 products of an exact
// three-way bf16 split (24 bits = 3 x 8; the dropped products are below 2^-24).
// The tensor pipe adds into its fp32 accumulators by truncation.  The corrections are
// 2^-8 (bf16) or 2^-11 (TF32) of the sum and have an accumulator set of their own, where
// their chain costs nothing; the leading products are a sixth or a third of the updates
// and, where their chain would still be long, dealt out over several sets.  The epilogue
// adds the sets, rounding to nearest.
//
// The output is swept along its slowest spatial dimension (S; D of a volume, H
// of an image).  A column holds TH rows (R) of 128 outputs (W), with as many
// output planes live as a staged plane reaches; a staged row feeds all live
// (row, plane) blocks at once, concatenated along N (3 x 3 taps x 16 filters:
// N = 144).  N is what makes the tensor pipe efficient here: an instruction
// takes max(N / 2, 32 + N / 4, 45) clocks (measured; the second term is the
// shared-memory read of A and B).  Which block a tap lands in rotates with the
// plane, so the filter image exists once per phase; images that do not fit stay
// in global memory and are streamed a plane ahead.
//
// Everything that depends on strides, paddings, phases and the direction of the
// pass is in tables built once on the host (conv_tc_shift.cu): per (phase, row)
// the accumulator ranges to update, per range the k-steps.  Backward data is the
// same machine on dy: with stride s the s x s x s input cells around an output
// position are one "super" position, whose sub-blocks each see their own taps.
//
// Warps: SH_EPI epilogue (two per TMEM lane quadrant), SH_CONV converters,
// SH_ISS MMA issuers (one thread each, rows dealt out in turn), one filter-image
// loader.  One thread can issue as fast as the tensor pipe takes instructions,
// but a row's waits, table reads and commits are a chain of some hundred
// dependent instructions: with few k-steps per row (four channels: five) they
// take longer than its products, so three rows are in issue at once.  Warps of
// one role share a scheduler as far as they can (warp & 3: the issuers and the
// loader on one, the converters on the other three, the epilogue on all four by
// its lane quadrants): what a scheduler's instruction cache has to hold is then
// two roles instead of four.
#pragma once

#include "conv_tc_common.cuh"

namespace dcb
{

constexpr int SH_EPI = 8;
constexpr int SH_CONV = 12;
constexpr int SH_ISS = 3;
constexpr int SH_THREADS = (SH_EPI + SH_CONV + SH_ISS + 1) * 32;
constexpr int SH_MAX_ITEMS = SH_CONV; // warp-sized pieces of a staged row: never more than the warps of a team
constexpr int SH_MAX_SLOTS = 9;   // A slots: a multiple of SH_ISS
constexpr int SH_MAX_BLOCKS = 64; // (row, plane slot) accumulator blocks of a column
// the epilogue's teams take blocks in turn; the same with statistics of the output; they share every block
constexpr int SH_PLAIN = 0, SH_STATS = 1, SH_SHARED = 2;

struct ShGroup // one accumulator range of a staged row
{
    uint16_t dcol, n;    // first TMEM column, width
    uint16_t step0, nst; // its k-steps
    uint32_t b16;        // filter image, 16-byte units from the start of its set
    uint32_t pad_;
};

// The issuers' tables (steps, groups, rows: offsets in ShGeom), in the constant bank.  What an
// instruction needs is then in uniform registers, where it has to be: alone on its SM, a warp
// issues an instruction every 45 clocks (N = 48), every 69 with the tables in shared memory, and
// beside the converters' traffic the difference grows.  16 -> 32, stride 2, 256^3 1048 -> 910 us,
// 16 -> 4 channels (backward data) 905 -> 868, 32 -> 32, 5 x 5 943 -> 901.  They are an argument of
// their own size class: 8 KB with every launch made passes of 30 us, which wait for the host, 3 %
// slower; the tables of most small layers fit 1 KB.
constexpr int SH_CONST = 8192, SH_CONST_SMALL = 1024;
template <int BYTES>
struct ShConst
{
    uint4 v[BYTES / 16];
};

// Spatial triples are in sweep terms: S (slowest), R, W.  "Super" output
// positions are outputs (forward) or s-cell groups of the input (backward data).
struct ShGeom
{
    int n, cin, kout;
    int in_s, in_r, in_w; // staged tensor
    long long xs_n, xs_c, xs_s, xs_r;
    int q_s, q_r, q_w; // super output extents
    int o_s, o_r, o_w; // output tensor
    long long ys_n, ys_c, ys_s, ys_r;
    int st_s, st_r, st_w;    // staged index = super * st + tap - pad
    int e_s, e_r, e_w;       // cells of a super position
    int fs, fr;              // taps of a super position in staged terms
    int pad_s, pad_r, pad_w;
    int th, rows;            // super rows of a column, staged rows of a plane
    int ns, nph;             // plane slots, phases
    int nb, kcols, kgroups;  // columns per cell block, filters per group
    int blk, rowst, woff, nsets, set_off; // columns: block, row of blocks, cell parity along W, set
    int cpg, cgroups;        // channels per group (a multiple of the cell's)
    int pt;                  // positions per plane of the A slot
    int ipr;                 // items (32 positions, all cells of the channel group) of a staged row
    int a_slot16, a_slots;
    int teams;               // converter teams; a_slots is a multiple of it and of SH_ISS
    int npack, pack_s, pack_r; // sub-columns side by side in the 128 lanes, their distance in super units
    int tile_w;              // super positions of a sub-column
    int tiles_w, hblks, nsegs, seglen;
    unsigned units;
    int stream;              // filter images are streamed per (plane, channel group)
    int b_stage16;           // 16-byte units of a stage (stream) or of one channel group's images
    int nsteps, ngroups;
    uint32_t rnd_add, rnd_mask;
    // byte offsets in shared memory
    int stage;               // bytes per epilogue warp for bulk stores, 0: none
    int so_stage, so_a, so_sets, so_items, so_lanes, so_bars;
    int co_groups, co_rows; // in the constant tables, 16-byte and 4-byte units (the steps stand first)
    // byte offsets in the table buffer (same order), total to copy
    int tab_bytes;
};

struct ShUnit
{
    int n, kg, q0, q1, qb, zr0, zr1, nz, row0, ow0;
    int z_lo, z_hi; // planes with any staged cell
    int i_lo, i_hi; // rows with any staged cell
};

// Not inlined: several divisions, called at a handful of places once per unit.
static __host__ __device__ __noinline__ ShUnit sh_unit(const ShGeom& g, uint32_t u)
{
    ShUnit t;
    const uint32_t tw = u % (uint32_t) g.tiles_w;
    u /= (uint32_t) g.tiles_w;
    const uint32_t hb = u % (uint32_t) g.hblks;
    u /= (uint32_t) g.hblks;
    const uint32_t sg = u % (uint32_t) g.nsegs;
    u /= (uint32_t) g.nsegs;
    t.n = (int) (u % (uint32_t) g.n);
    t.kg = (int) (u / (uint32_t) g.n);
    const int sub_s = g.pack_s > 0 ? g.npack : 1, sub_r = g.pack_r > 0 ? g.npack : 1;
    t.q0 = (int) sg * g.seglen * sub_s;
    t.q1 = min(t.q0 + g.seglen, g.q_s);
    t.row0 = (int) hb * g.th * sub_r;
    t.ow0 = (int) tw * g.tile_w;
    const int reach = (g.fs - 1) / g.st_s;
    t.qb = t.q0 - reach;
    t.zr0 = (t.q0 - t.qb) * g.st_s;
    t.zr1 = (t.q1 - 1 - t.qb) * g.st_s + g.fs;
    t.nz = (t.q1 - 1 - t.qb + reach) * g.st_s + g.fs;
    // staged plane index of step z: qb * st + z - pad (+ the sub-column's distance)
    const int p0 = t.qb * g.st_s - g.pad_s;
    const int far = (sub_s - 1) * g.pack_s * g.st_s;
    t.z_lo = max(t.zr0, -(p0 + far));
    t.z_hi = min(t.zr1, g.in_s - p0);
    const int r0 = t.row0 * g.st_r - g.pad_r;
    t.i_lo = sub_r > 1 ? 0 : max(0, -r0);
    t.i_hi = min(g.rows, g.in_r - r0);
    if (t.i_hi <= t.i_lo)
        t.z_hi = t.z_lo;
    return t;
}

__device__ __forceinline__ uint32_t pack_hi16(uint32_t lo, uint32_t hi)
{
    return __byte_perm(lo, hi, 0x7632); // upper halves of both
}

// D += A * B, issued by the elected lane of a converged warp.  No memory clobber:
// the tables that the next steps come from may be read ahead; order among the
// instruction, the waits and the commits is kept by their being volatile.
template <int KIND>
__device__ __forceinline__ void sh_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t elected)
{
    if (KIND == 0)
        asm volatile("{\n\t.reg .pred e, t;\n\tsetp.ne.b32 e, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
                     "@e tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, t;\n\t}" ::"r"(d),
                     "l"(a), "l"(b), "r"(idesc), "r"(elected));
    else
        asm volatile("{\n\t.reg .pred e, t;\n\tsetp.ne.b32 e, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
                     "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, t;\n\t}" ::"r"(d),
                     "l"(a), "l"(b), "r"(idesc), "r"(elected));
}

__device__ __forceinline__ uint32_t elect_one()
{
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e;
}

// One cell (4 or 8 channels of one position) split into PARTS operands and
// stored `part_stride` bytes apart.
template <int KIND, int PARTS>
__device__ __forceinline__ void sh_convert_store(const float (&v)[KIND == 0 ? 4 : 8], uint32_t dst,
                                                 uint32_t part_stride, uint32_t rnd_add, uint32_t rnd_mask)
{
    constexpr int CH = KIND == 0 ? 4 : 8;
    uint32_t w[PARTS][4];
    if (KIND == 0)
    {
#pragma unroll
        for (int c = 0; c < CH; ++c)
        {
            const uint32_t hi = (PARTS == 1 ? round_fast(v[c], rnd_add) : __float_as_uint(v[c]) + rnd_add) & rnd_mask;
            w[0][c & 3] = hi;
            if (PARTS > 1) // exact remainder below 2^-11 |x| (or not a number); the pipe reads its upper 19 bits
                w[PARTS - 1][c & 3] = __float_as_uint(v[c] - __uint_as_float(hi));
        }
    }
    else if (PARTS == 1)
    {
#pragma unroll
        for (int c = 0; c < CH; c += 2)
            w[0][c / 2] = pack_hi16(round_fast(v[c], rnd_add), round_fast(v[c + 1 < CH ? c + 1 : c], rnd_add));
    }
    else
    {
        // truncating split: 8 + 8 + 8 significant bits, nothing is lost
        float r[CH], q[CH];
#pragma unroll
        for (int c = 0; c < CH; ++c)
        {
            r[c] = v[c] - __uint_as_float(__float_as_uint(v[c]) & 0xffff0000u);
            q[c] = r[c] - __uint_as_float(__float_as_uint(r[c]) & 0xffff0000u);
        }
#pragma unroll
        for (int c = 0; c < CH; c += 2)
        {
            const int d = c + 1 < CH ? c + 1 : c;
            w[0][c / 2] = pack_hi16(__float_as_uint(v[c]), __float_as_uint(v[d]));
            w[PARTS > 1 ? 1 : 0][c / 2] = pack_hi16(__float_as_uint(r[c]), __float_as_uint(r[d]));
            w[PARTS - 1][c / 2] = pack_hi16(__float_as_uint(q[c]), __float_as_uint(q[d]));
        }
    }
#pragma unroll
    for (int p = 0; p < PARTS; ++p)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + (uint32_t) p * part_stride), "r"(w[p][0]),
                     "r"(w[p][1]), "r"(w[p][2]), "r"(w[p][3])
                     : "memory");
}

// Position of a warp in the sequence of staged rows of its CTA (rows and planes
// without any cell of the tensor are left out; the issuers leave them out too).
struct ShCursor
{
    ShUnit u;
    uint32_t unit;
    int z, grp, i;
    uint32_t slot, lap; // ring slot of the row, how often the ring has gone round
    bool live;

    __device__ __forceinline__ void first(const ShGeom& g, int rows)
    {
        unit = blockIdx.x;
        slot = 0;
        lap = 0;
        live = true;
        enter(g);
        advance(g, rows);
    }
    __device__ __forceinline__ void enter(const ShGeom& g)
    {
#pragma unroll 1
        for (; unit < g.units; unit += gridDim.x)
        {
            u = sh_unit(g, unit);
            if (u.z_hi > u.z_lo)
            {
                z = u.z_lo;
                grp = 0;
                i = u.i_lo;
                return;
            }
        }
        live = false;
    }
    __device__ __forceinline__ void advance(const ShGeom& g, int rows)
    {
        slot += (uint32_t) rows;
#pragma unroll 1
        while (slot >= (uint32_t) g.a_slots)
        {
            slot -= (uint32_t) g.a_slots;
            ++lap;
        }
        i += rows;
#pragma unroll 1
        while (live && i >= u.i_hi)
        {
            const int over = i - u.i_hi;
            if (++grp == g.cgroups)
            {
                grp = 0;
                if (++z == u.z_hi)
                {
                    unit += gridDim.x;
                    enter(g);
                }
            }
            i = u.i_lo + over;
        }
    }
};

// What a product is of, for the outputs whose accumulators are no numbers.  Spatial triples are
// in sweep terms, as in ShGeom.
struct ShExact
{
    const float *x, *w; // (the kernel's own x occupies registers, here it is a constant)
    float alpha;
    const uint32_t* w_flag; // holds `call` if the filter of this call has an element that is no number
    uint32_t* out_flag;     // ... if an output may be none
    uint32_t call;
    int transposed, one_pass;
    int f[3], stride[3], pad[3];
    long long w_ko, w_ci;
};

// An infinity has no second part (inf - inf), and an instruction also multiplies it with the
// zeros that stand for taps an output does not have: either leaves a NaN where there may be a
// number or an infinity.  So one output by FMAs over its taps, as the CUDA-core kernels do it.
__device__ __noinline__ static float sh_exact(const ShGeom& g, const ShExact& e, int n, int ko, int os, int orow, int ow)
{
    float acc = 0.f;
    auto staged = [&](int d, int o, int k, int extent) { // staged index of tap k, or -1
        int i = e.transposed ? o + e.pad[d] - k : o * e.stride[d] + k - e.pad[d];
        if (e.transposed)
            i = i >= 0 && i % e.stride[d] == 0 ? i / e.stride[d] : -1;
        return i < extent ? i : -1;
    };
    for (int ks = 0; ks < e.f[0]; ++ks)
    {
        const int is = staged(0, os, ks, g.in_s);
        if (is < 0)
            continue;
        for (int kr = 0; kr < e.f[1]; ++kr)
        {
            const int ir = staged(1, orow, kr, g.in_r);
            if (ir < 0)
                continue;
            for (int kw = 0; kw < e.f[2]; ++kw)
            {
                const int iw = staged(2, ow, kw, g.in_w);
                if (iw < 0)
                    continue;
                const float* xp = e.x + (long long) n * g.xs_n + (long long) is * g.xs_s + (long long) ir * g.xs_r + iw;
                const float* wp = e.w + (long long) ko * e.w_ko + (ks * e.f[1] + kr) * e.f[2] + kw;
                for (int c = 0; c < g.cin; ++c)
                {
                    float a = xp[(long long) c * g.xs_c], b = wp[(long long) c * e.w_ci];
                    if (e.one_pass)
                    {
                        a = __uint_as_float(round_operand(a, g.rnd_add, g.rnd_mask));
                        b = __uint_as_float(round_operand(e.alpha * b, g.rnd_add, g.rnd_mask));
                    }
                    acc = fmaf(a, b, acc);
                    if (acc != acc)
                        return acc; // and stays that
                }
            }
        }
    }
    return e.one_pass ? acc : e.alpha * acc;
}

// Columns of tensor memory that the epilogue may fetch: 16 at a time, also where fewer are left of
// the last block.  What it fetches it may look at, so all of them are zeroed first.  (With only the
// accumulators' columns zeroed, backward data of 4 channels on 64 x 128 x 128, stride 2 along D and
// W, took what an earlier kernel had left beyond them for outputs that are no numbers and went to
// look for those: 112 us behind a kernel of NaNs, 77 behind others; 79 and 77 like this.)
__host__ __device__ __forceinline__ int sh_columns(const ShGeom& g)
{
    return g.set_off * g.nsets + (g.nb % 16 ? 16 - g.nb % 16 : 0);
}

// Columns without a spare plane slot, of one row: a block has to be drained before its slot is
// opened again, by the next plane, so that nothing else goes on meanwhile. Both epilogue teams
// then share every block where it has two halves (cells of either parity along W, or pieces of 16
// filters): 32 -> 16, stride 2, backward data on 256^3 944 -> 804 us, 24 -> 28 forward on 40 x 100 x 132
// 311 -> 300. (A kernel of its own: with the choice at run time all others lost 1 %.)
inline bool sh_shared_drain(const ShGeom& g)
{
    return g.th == 1 && g.ns * g.st_s < g.fs + g.st_s && (g.e_w == 2 || (g.e_s * g.e_r == 1 && g.nb > 16));
}

// An issuer reports a block as complete when its next row, SH_ISS further on, is past the block's last one. Where
// a plane's blocks are opened and closed in the same step (one tap along the sweep), those are only the
// blocks up to its own row: it has waited for no others to be free, and a report of one that is still in
// use counts for that use.
__host__ __device__ __forceinline__ int sh_reports_ahead(const ShGeom& g)
{
    return g.fs > 1 ? SH_ISS : min(SH_ISS, g.fr);
}

__device__ __forceinline__ bool sh_number(float v)
{
    return fabsf(v) <= 3.402823466e+38f;
}

// Goes through the outputs of this CTA's units once more and computes those that are no numbers
// by themselves; then the statistics, if there are any, from what stands there.  After the
// kernel's last barrier, by all threads; not for beta != 0, where the old output is gone.
template <bool STATS>
__device__ __noinline__ static void sh_repair(const ShGeom& g, const ShExact& ex, float* y, float* stat_part)
{
    const int cells = g.e_s * g.e_r * g.e_w, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int subs_s = g.pack_s > 0 ? g.npack : 1, subs_r = g.pack_r > 0 ? g.npack : 1;
    float st1 = 0.f, st2 = 0.f; // of filter `warp`
    asm volatile("fence.proxy.async;" ::: "memory"); // bulk stores before plain loads
    for (int pass = 0; pass < (STATS ? 2 : 1); ++pass)
    {
#pragma unroll 1
        for (uint32_t unit = blockIdx.x; unit < g.units; unit += gridDim.x)
        {
            const ShUnit u = sh_unit(g, unit);
            const int kbase = u.kg * g.kcols, kn = min(g.kcols, g.kout - kbase), planes = u.q1 - u.q0;
            const long long rows = (long long) planes * subs_s * g.th * subs_r;
#pragma unroll 1
            for (long long row = pass == 0 ? warp : 0; row < rows; row += pass == 0 ? SH_THREADS / 32 : 1)
            {
                // (sub-column, plane, sub-column, row)
                const int r = u.row0 + (int) (row % g.th) + (int) (row / g.th % subs_r) * g.pack_r;
                const int q = u.q0 + (int) (row / g.th / subs_r % planes) + (int) (row / g.th / subs_r / planes) * g.pack_s;
                if (r >= g.q_r || q >= g.q_s)
                    continue;
#pragma unroll 1
                for (int i = lane; i < g.tile_w * cells; i += 32)
                {
                    const int qw = u.ow0 + i / cells, cell = i % cells;
                    const int os = q * g.e_s + cell / (g.e_r * g.e_w), orow = r * g.e_r + cell / g.e_w % g.e_r, ow = qw * g.e_w + cell % g.e_w;
                    if (qw >= g.q_w || os >= g.o_s || orow >= g.o_r || ow >= g.o_w)
                        continue;
                    float* yp = y + (long long) u.n * g.ys_n + (long long) kbase * g.ys_c + (long long) os * g.ys_s
                                + (long long) orow * g.ys_r + ow;
                    if (pass == 0)
                    {
#pragma unroll 1
                        for (int k = 0; k < kn; ++k)
                            if (!sh_number(yp[k * g.ys_c]))
                                yp[k * g.ys_c] = sh_exact(g, ex, u.n, kbase + k, os, orow, ow);
                    }
                    else if (warp < kn)
                    {
                        const float v = yp[warp * g.ys_c];
                        st1 += v;
                        st2 = fmaf(v, v, st2);
                    }
                }
            }
        }
        __syncthreads();
    }
    if (STATS && warp < 16)
    {
        for (int o = 16; o > 0; o >>= 1)
        {
            st1 += __shfl_xor_sync(0xffffffffu, st1, o);
            st2 += __shfl_xor_sync(0xffffffffu, st2, o);
        }
        for (int w = lane; w < SH_EPI; w += 32) // the epilogue warps' partials
        {
            float* part = stat_part + ((size_t) blockIdx.x * SH_EPI + w) * 32;
            part[warp] = w == 0 ? st1 : 0.f;
            part[16 + warp] = w == 0 ? st2 : 0.f;
        }
    }
}

// A value that all lanes of a converged warp have, where the compiler does not know it.
__device__ __forceinline__ uint32_t uniform(uint32_t v)
{
    return __shfl_sync(0xffffffffu, v, 0);
}

// A wait may end for one lane as it runs out for another: the warp stays together.
__device__ __forceinline__ bool all_lanes(bool ok)
{
    return __all_sync(0xffffffffu, ok) != 0;
}

// Keeps a uniform condition inside its loop: hoisted out, every such condition
// doubles the loop, and the roles of this kernel share one instruction cache
// (95 KB of code ran four times slower than 30 KB).
__device__ __forceinline__ int in_loop(int v)
{
    asm volatile("" : "+r"(v));
    return v;
}

__device__ __forceinline__ void sh_tmem_ld16(uint32_t taddr, uint32_t (&v)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(taddr));
}

__device__ __forceinline__ void sh_tmem_zero(uint32_t taddr, int n)
{
    if (in_loop(n) >= 16)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
                     "{%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr),
                     "r"(0u)
                     : "memory");
    else
#pragma unroll 1
        for (int c = 0; c < n; c += 4)
            asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %1, %1, %1};" ::"r"(taddr + (uint32_t) c),
                         "r"(0u)
                         : "memory");
}

// The registers of a tensor-memory load may be read after this.
__device__ __forceinline__ void sh_loaded(uint32_t (&v)[16])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                   "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])
                 :
                 : "memory");
}

// Up to 16 accumulator columns of this warp's lanes: fetched (always 16, the
// columns past n belong to other blocks and are ignored), summed over the sets,
// zeroed in tensor memory.  A load takes some thousand clocks with products in
// flight: those of the first two sets are on their way together.
__device__ __forceinline__ void sh_drain(uint32_t taddr, int n, int nsets, int set_off, float (&v)[16])
{
    uint32_t a[16];
    sh_tmem_ld16(taddr, a);
    if (in_loop(nsets) > 1)
    {
        uint32_t b[16];
        uint32_t set = taddr + (uint32_t) set_off;
        sh_tmem_ld16(set, b);
        sh_loaded(a);
        sh_loaded(b);
#pragma unroll
        for (int k = 0; k < 16; ++k)
            v[k] = __uint_as_float(a[k]) + __uint_as_float(b[k]);
        sh_tmem_zero(set, n);
#pragma unroll 1
        for (int s = 2; s < in_loop(nsets); ++s)
        {
            set += (uint32_t) set_off;
            sh_tmem_ld16(set, b);
            sh_loaded(b);
#pragma unroll
            for (int k = 0; k < 16; ++k)
                v[k] += __uint_as_float(b[k]);
            sh_tmem_zero(set, n);
        }
    }
    else
    {
        sh_loaded(a);
#pragma unroll
        for (int k = 0; k < 16; ++k)
            v[k] = __uint_as_float(a[k]);
    }
    sh_tmem_zero(taddr, n);
}

// Up to 16 filters of one output position, ys_c elements apart.
__device__ __forceinline__ void sh_store(float* p, long long ys_c, int n, float beta, float (&v)[16])
{
    if (__int_as_float(in_loop(__float_as_int(beta))) != 0.f)
    {
        const float* o = p;
#pragma unroll
        for (int k = 0; k < 16; ++k, o += ys_c)
            v[k] = k < n ? fmaf(beta, *o, v[k]) : 0.f;
    }
    if (in_loop(n) >= 16)
    {
#pragma unroll
        for (int k = 0; k < 16; ++k, p += ys_c)
            *p = v[k];
        return;
    }
#pragma unroll
    for (int k = 0; k < 16; ++k, p += ys_c)
        if (k < n)
            *p = v[k];
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}


// WIDE: channels lie too far apart for 32-bit offsets.  (64-bit offsets throughout, or two
// pointers per channel pair, make every other layer 1 to 2 % slower.)
template <int KIND, int PARTS, int EPILOGUE, bool WIDE, int CONST>
__global__ void __launch_bounds__(SH_THREADS, 1)
    sh_conv_kernel(const __grid_constant__ ShGeom g, const __grid_constant__ ShExact ex, float beta, const __grid_constant__ ShConst<CONST> ct,
                   const float* __restrict__ x, const uint4* __restrict__ bimg, const uint8_t* __restrict__ tables, float* y, int* status,
                   float* __restrict__ stat_part, const __grid_constant__ CUtensorMap ymap, int use_ymap)
{
    constexpr int CH = KIND == 0 ? 4 : 8;
    constexpr bool STATS = EPILOGUE == SH_STATS, SHARED = EPILOGUE == SH_SHARED;
    constexpr int HALVES = SHARED ? 2 : 1;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    const uint2* sets = reinterpret_cast<const uint2*>(smem + g.so_sets);
    const uint32_t* items = reinterpret_cast<const uint32_t*>(smem + g.so_items);
    const int* lanes = reinterpret_cast<const int*>(smem + g.so_lanes);
    uint64_t* a_full = reinterpret_cast<uint64_t*>(smem + g.so_bars); // [a_slots] converters -> issuer
    uint64_t* a_empty = a_full + g.a_slots;                           // [a_slots] issuer -> converters
    uint64_t* b_full = a_empty + g.a_slots;                           // [2] loader -> issuer
    uint64_t* b_empty = b_full + 2;                                   // [2] issuer -> loader
    uint64_t* ev_full = b_empty + 2;                                  // [th * ns] issuer -> epilogue: block complete
    uint64_t* ev_empty = ev_full + g.th * g.ns;                       // [th * ns] epilogue -> issuer: block zeroed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ev_empty + g.th * g.ns);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // roles: warps 0..7 epilogue; of the others, every fourth an issuer and the last of those the loader
    const int turn_w = (warp - SH_EPI) >> 2;
    const bool is_conv = warp >= SH_EPI && (warp & 3) != 3;
    const int conv_w = turn_w * 3 + (warp & 3), iss_w = turn_w;

    // A small layer is one pass through this set-up: a thread per barrier (64 blocks at most)
    static_assert(SH_MAX_SLOTS <= 32 && SH_MAX_BLOCKS <= 64, "a warp's lanes");
    if (warp == 1)
    {
        if (lane < g.a_slots)
        {
            mbar_init(&a_full[lane], (uint32_t) g.ipr);
            mbar_init(&a_empty[lane], 1);
        }
        if (lane < 2)
        {
            mbar_init(&b_full[lane], 1);
            mbar_init(&b_empty[lane], SH_ISS);
        }
#pragma unroll 1
        for (int b = lane; b < g.th * g.ns; b += 32)
        {
            mbar_init(&ev_full[b], SH_ISS);
            mbar_init(&ev_empty[b], SHARED ? SH_EPI : 4);
        }
        if (lane == 0)
        {
            *abort_flag = 0;
            abort_flag[1] = 0; // an output that is no number
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0)
    {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(TC_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
#pragma unroll 1
    for (int i = tid; i < g.tab_bytes / 16; i += SH_THREADS)
        reinterpret_cast<uint4*>(smem + g.so_sets)[i] = reinterpret_cast<const uint4*>(tables)[i];
    // positions that no item writes are read by the MMAs of lanes nobody stores: keep them finite
#pragma unroll 1
    for (int i = tid; i < g.a_slots * g.a_slot16; i += SH_THREADS)
        reinterpret_cast<uint4*>(smem + g.so_a)[i] = make_uint4(0, 0, 0, 0);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (warp < SH_EPI)
#pragma unroll 1
        for (int c = (warp >> 2) * 16; c < sh_columns(g); c += 32)
            sh_tmem_zero(tmem_base + ((uint32_t) ((warp & 3) * 32) << 16) + (uint32_t) c, 16);
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // the filter image, the input and everything that is written
    wait_for_previous_kernel(x);
    bool ok = true;

    if (warp < SH_EPI)
    {
        // ------------------------------------------------------------------
        // epilogue: blocks complete in (plane, row) order; the teams take them
        // in turn.  The same block comes round every th * ns blocks; there
        // are never more teams than that, so a team that has seen the block
        // before its own complete knows that the previous use of its block is
        // complete too, and the parity it waits on cannot be two uses behind.
        // ------------------------------------------------------------------
        const int quad = warp & 3, team = warp >> 2;
        const int teams = min(SH_EPI / 4, g.th * g.ns);
        const uint32_t lane_addr = tmem_base + ((uint32_t) (quad * 32) << 16);
        const int lt = lanes[quad * 32 + lane];
        const int sub = lt >> 16, xx = lt & 0xffff;
        const bool lane_on = lt >= 0 && xx < g.tile_w;
        const int add_s = sub * g.pack_s, add_r = sub * g.pack_r;
        float st1[STATS ? 16 : 1], st2[STATS ? 16 : 1];
#pragma unroll
        for (int k = 0; k < (STATS ? 16 : 1); ++k)
            st1[k] = st2[k] = 0.f;
        uint32_t slot = 0, lap = 0; // plane slot of the block, uses of it before
        // An element of x that is no number makes one of every filter's sum (times zero too): the
        // first filter of a fetch shows it.  Elements of w are looked at when they are packed.
        bool numbers = true;
        const uint32_t stage_s = smem_u32(smem + g.so_stage) + (uint32_t) (warp * g.stage);
        const uint32_t stage_lane = stage_s + 4u * lane;
        const bool store_w = quad * 32 < g.tile_w;
        static_assert(SH_EPI == 8, "two teams, a half each");
        const int half = SHARED ? team : 0; // of every block
        int j = SHARED ? 0 : team < teams ? team : 0x40000000;
#pragma unroll 1
        for (uint32_t unit = blockIdx.x; unit < g.units && ok; unit += gridDim.x)
        {
            const ShUnit u = sh_unit(g, unit);
            const int nq = (u.nz - g.fs) / g.st_s + 1;
            const int kbase = u.kg * g.kcols, kn = min(g.kcols, g.kout - kbase);
            const int qw = u.ow0 + xx;
            const bool lane_w = lane_on && qw < g.q_w;
#pragma unroll 1
            for (int qi = 0; qi < nq && ok; ++qi)
            {
                const bool live = u.qb + qi >= u.q0 && u.qb + qi < u.q1;
                const int q = u.qb + qi + add_s;
                // this team's blocks of the plane; the count goes on into the next one
#pragma unroll 1
                for (; j < g.th; j += SHARED ? 1 : teams)
                {
                    const int b = j * g.ns + (int) slot;
                    ok = mbar_wait(&ev_full[b], lap & 1, abort_flag);
                    if (!ok)
                        break;
                    tc_fence_after();
                    const int r = u.row0 + j + add_r;
                    const bool on = lane_w && live && q < g.q_s && r < g.q_r;
                    const uint32_t block = lane_addr + (uint32_t) (j * g.rowst + (int) slot * g.blk);
                    if (!SHARED && use_ymap)
                    {
                        // one bulk tensor store per warp: 32 positions of every filter
                        float v[16];
                        sh_drain(block, g.nb, g.nsets, g.set_off, v);
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0)
                            mbar_arrive(&ev_empty[b]);
                        if (!live || r >= g.q_r || !store_w)
                            continue;
                        numbers = numbers && sh_number(v[0]);
                        if (STATS && lane_w)
                        {
#pragma unroll
                            for (int k = 0; k < (STATS ? 16 : 0); ++k)
                            {
                                st1[k] += v[k];
                                st2[k] = fmaf(v[k], v[k], st2[k]);
                            }
                        }
                        // (the buffer's previous store has been read)
                        if (lane == 0)
                            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                        __syncwarp();
#pragma unroll
                        for (int k = 0; k < 16; ++k)
                            asm volatile("st.shared.f32 [%0], %1;" ::"r"(stage_lane + 128u * k), "f"(v[k]) : "memory");
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                        if (lane == 0)
                        {
                            asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.tile.bulk_group "
                                         "[%0, {%2, %3, %4, %5, %6}], [%1];" ::"l"(reinterpret_cast<uint64_t>(&ymap)),
                                         "r"(stage_s), "r"(u.ow0 + quad * 32), "r"(r), "r"(q), "r"(kbase), "r"(u.n)
                                         : "memory");
                            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                        }
                        continue;
                    }
                    float* yp = y + (long long) u.n * g.ys_n + (long long) kbase * g.ys_c;
                    if (STATS || g.e_s * g.e_r * g.e_w == 1)
                    {
                        yp += (long long) q * g.ys_s + (long long) r * g.ys_r + qw;
#pragma unroll 1
                        for (int k0 = 16 * half; k0 < in_loop(g.nb); k0 += 16 * HALVES)
                        {
                            float v[16];
                            const int piece = min(16, g.nb - k0);
                            sh_drain(block + (uint32_t) k0, piece, g.nsets, g.set_off, v);
                            if (k0 + 16 * HALVES >= g.nb)
                            {
                                // last columns of the block: hand it back before the stores
                                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                                tc_fence_before();
                                __syncwarp();
                                if (lane == 0)
                                    mbar_arrive(&ev_empty[b]);
                            }
                            numbers = numbers && sh_number(v[0]);
                            if (STATS && in_loop(on))
                            {
                                // (columns past the filters hold zeros or are not folded)
#pragma unroll
                                for (int k = 0; k < (STATS ? 16 : 0); ++k)
                                {
                                    st1[k] += v[k];
                                    st2[k] = fmaf(v[k], v[k], st2[k]);
                                }
                            }
                            if (in_loop(on))
                                sh_store(yp + (long long) k0 * g.ys_c, g.ys_c, min(piece, kn - k0), beta, v);
                        }
                        continue;
                    }
                    if (in_loop(g.nb) < 16)
                    {
                        // Cells of the same parity along W lie side by side: a fetch of 16 columns
                        // is four quarters, each of one cell (4 -> 16, stride 2, 64 x 128 x 128: 79 us
                        // with a fetch per cell, 48 like this; of 16 filters 992 per cell, 1275).
#pragma unroll 1
                        for (int ew = half; ew < in_loop(g.e_w); ew += HALVES)
                        {
                            const int ow = qw * g.e_w + ew, cols = g.e_s * g.e_r * g.nb;
                            int es = 0, er = 0, k0 = 0; // of the next quarter
#pragma unroll 1
                            for (int c0 = 0; c0 < in_loop(cols); c0 += 16)
                            {
                                float v[16];
                                sh_drain(block + (uint32_t) (ew * g.woff + c0), min(16, cols - c0), g.nsets, g.set_off, v);
                                numbers = numbers && sh_number(v[0]) && sh_number(v[4]) && sh_number(v[8]) && sh_number(v[12]);
#pragma unroll
                                for (int h = 0; h < 4; ++h)
                                {
                                    const int os = q * g.e_s + es, orow = r * g.e_r + er;
                                    const bool put = on && es < g.e_s && os < g.o_s && orow < g.o_r && ow < g.o_w;
                                    float* yc = yp + (long long) os * g.ys_s + (long long) orow * g.ys_r + ow + (long long) k0 * g.ys_c;
#pragma unroll
                                    for (int k = 0; k < 4; ++k, yc += g.ys_c)
                                        if (put && k0 + k < kn)
                                            *yc = beta != 0.f ? fmaf(beta, *yc, v[4 * h + k]) : v[4 * h + k];
                                    k0 += 4;
                                    if (k0 >= g.nb)
                                    {
                                        k0 = 0;
                                        if (++er == g.e_r)
                                            er = 0, ++es;
                                    }
                                }
                            }
                        }
                    }
                    else
#pragma unroll 1
                        for (int es = 0; es < in_loop(g.e_s); ++es)
#pragma unroll 1
                            for (int er = 0; er < in_loop(g.e_r); ++er)
#pragma unroll 1
                                for (int ew = half; ew < in_loop(g.e_w); ew += HALVES)
                                {
                                    const uint32_t cell = block + (uint32_t) (ew * g.woff + (es * g.e_r + er) * g.nb);
                                    const int os = q * g.e_s + es, orow = r * g.e_r + er, ow = qw * g.e_w + ew;
                                    const bool put = on && os < g.o_s && orow < g.o_r && ow < g.o_w;
                                    float* yc = yp + (long long) os * g.ys_s + (long long) orow * g.ys_r + ow;
#pragma unroll 1
                                    for (int k0 = 0; k0 < in_loop(g.nb); k0 += 16)
                                    {
                                        float v[16];
                                        const int piece = min(16, g.nb - k0);
                                        sh_drain(cell + (uint32_t) k0, piece, g.nsets, g.set_off, v);
                                        numbers = numbers && sh_number(v[0]);
                                        if (in_loop(put))
                                            sh_store(yc + (long long) k0 * g.ys_c, g.ys_c, min(piece, kn - k0), beta, v);
                                    }
                                }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(&ev_empty[b]);
                }
                j -= g.th;
                if (++slot == (uint32_t) g.ns)
                {
                    slot = 0;
                    ++lap;
                }
            }
        }
        if (!numbers)
            abort_flag[1] = 1;
        if (use_ymap && lane == 0)
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        if (STATS)
        {
            // this warp's partials: 16 sums, 16 sums of squares over its lanes
#pragma unroll
            for (int k = 0; k < 16; ++k)
            {
                float a = st1[STATS ? k : 0], b = st2[STATS ? k : 0];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                {
                    a += __shfl_xor_sync(0xffffffffu, a, o);
                    b += __shfl_xor_sync(0xffffffffu, b, o);
                }
                if (lane == 0)
                {
                    float* part = stat_part + ((size_t) blockIdx.x * SH_EPI + warp) * 32;
                    part[k] = a;
                    part[16 + k] = b;
                }
            }
        }
    }
    else if (is_conv)
    {
        // ------------------------------------------------------------------
        // converters: a staged row is g.ipr items of 32 positions.  A team of
        // g.ipr warps converts a row, each always the same positions, so that
        // what a row costs is its cells; the teams take rows in turn (a slot is
        // only ever one team's, so its release is never two laps away).  Loads
        // run two cells ahead.
        // ------------------------------------------------------------------
        const int teams = g.teams, team = conv_w / g.ipr;
        const uint32_t it = items[conv_w % g.ipr];
        const int par = (int) (it & 255u), pos = (int) (it >> 8) + lane;
        const int lt = lanes[pos];
        const int sub = max(lt, 0) >> 16, xx = max(lt, 0) & 0xffff;
        // staged cell of this lane relative to the row's first: in bytes, for the channels
        // of a cell (WIDE: for one channel); planes and rows are added to the base pointers
        uint32_t off[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
            off[e] = 4u * (uint32_t) (xx * g.st_w + par + sub * (g.pack_s * g.st_s * (int) g.xs_s + g.pack_r * g.st_r * (int) g.xs_r)
                                      + (WIDE ? 0 : e * (int) g.xs_c));
        const uint32_t dpos = lt >= 0 ? smem_u32(smem + g.so_a) + 16u * (uint32_t) (par * g.pt + pos) : 0u;
        const uint32_t part_stride = (uint32_t) g.a_slot16 / PARTS * 16u;
        const uint32_t cell_stride = (uint32_t) (g.st_w * g.pt) * 16u;
        const uint32_t full_s = smem_u32(a_full), empty_s = smem_u32(a_empty);
        const int cells = g.cpg / CH;
        ShCursor c;
        if (team < teams)
            c.first(g, team);
        float v[2][CH];
        uint32_t dst[2] = {0, 0};  // where the cell goes
        uint32_t wait[2] = {0, 0}; // barrier to wait for first | parity (0: none)
        uint32_t tell[2] = {0, 0}; // barrier to arrive on afterwards (0: none)
        bool has[2] = {false, false};
        bool more = team < teams, fresh = true; // fresh: the cursor has not moved off the first row yet
        int left = 0, nch = 0, nch0 = 0, row = 0;
        const char* row_p = reinterpret_cast<const char*>(x); // the row's first cell, channel 0
        const char* p = row_p;
        const long long row_step = 4ll * teams * g.xs_r, ch_step = 4ll * g.xs_c, ch4_step = 4 * ch_step;
        const uint32_t slot_bytes = 16u * (uint32_t) g.a_slot16;
        uint32_t d = 0;
        bool in = false, plane_in = false;
#pragma unroll 1
        while (ok && (more || has[0]))
        {
#pragma unroll
            for (int q = 0; q < 2; ++q)
            {
                if (has[q])
                {
                    if (wait[q] != 0)
                        ok = ok && mbar_wait_s<20>(wait[q] & ~7u, wait[q] & 1u, abort_flag);
                    if (dst[q] != 0)
                        sh_convert_store<KIND, PARTS>(v[q], dst[q], part_stride, g.rnd_add, g.rnd_mask);
                    if (tell[q] != 0)
                    {
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                        if (lane == 0)
                            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tell[q]) : "memory");
                    }
                }
                wait[q] = 0;
                if (left == 0 && more)
                {
                    if (!fresh && c.i + teams < c.u.i_hi)
                    {
                        // the team's next row of the same plane
                        c.i += teams;
                        row_p += row_step;
                        c.slot += (uint32_t) teams;
                        if (c.slot >= (uint32_t) g.a_slots)
                        {
                            c.slot -= (uint32_t) g.a_slots;
                            ++c.lap;
                        }
                    }
                    else
                    {
                        if (!fresh)
                            c.advance(g, teams);
                        fresh = false;
                        more = c.live;
                        const int s0 = c.u.qb * g.st_s + c.z - g.pad_s, r0 = c.u.row0 * g.st_r - g.pad_r,
                                  w0 = c.u.ow0 * g.st_w - g.pad_w;
                        row = r0 + sub * g.pack_r * g.st_r;
                        plane_in = lt >= 0 && (unsigned) (s0 + sub * g.pack_s * g.st_s) < (unsigned) g.in_s
                                   && (unsigned) (w0 + xx * g.st_w + par) < (unsigned) g.in_w;
                        row_p = reinterpret_cast<const char*>(
                            x + (long long) c.u.n * g.xs_n + (long long) (c.grp * g.cpg) * g.xs_c + (long long) s0 * g.xs_s
                            + (long long) (r0 + c.i) * g.xs_r + w0);
                        nch0 = g.cin - c.grp * g.cpg;
                    }
                    in = plane_in && (unsigned) (row + c.i) < (unsigned) g.in_r;
                    p = row_p;
                    nch = nch0;
                    d = dpos + c.slot * slot_bytes;
                    left = cells;
                    wait[q] = c.lap > 0 ? (empty_s + 8u * c.slot) | ((c.lap - 1) & 1u) : 0u;
                }
                has[q] = more;
                if (more)
                {
#pragma unroll
                    for (int e = 0; e < CH; ++e)
                        v[q][e] = 0.f;
                    if (in)
                    {
                        if (nch >= CH)
                        {
#pragma unroll
                            for (int e = 0; e < CH; ++e)
                                v[q][e] = __ldg(reinterpret_cast<const float*>((e < 4 ? p : p + ch4_step) + (WIDE ? (e & 3) * ch_step : 0) + off[e & 3]));
                        }
                        else
                        {
#pragma unroll
                            for (int e = 0; e < CH; ++e)
                                if (e < nch)
                                    v[q][e] = __ldg(reinterpret_cast<const float*>((e < 4 ? p : p + ch4_step) + (WIDE ? (e & 3) * ch_step : 0) + off[e & 3]));
                        }
                    }
                    p += CH / 4 * ch4_step;
                    nch -= CH;
                    dst[q] = dpos != 0 ? d : 0u;
                    d += cell_stride;
                    tell[q] = --left == 0 ? full_s + 8u * c.slot : 0u;
                }
            }
        }
    }
    else if (iss_w < SH_ISS)
    {
        // ------------------------------------------------------------------
        // issuers: the warp walks the sequence together, one lane issues.
        // Issuer w takes every SH_ISS-th staged row (A slots are dealt the same
        // way: a slot is only ever one issuer's).  Every issuer waits for every
        // block to be free and reports every block, so that no barrier can be
        // two completions away from a waiter.
        // ------------------------------------------------------------------
        const uint32_t elected = elect_one();
        const uint32_t a16 = smem_u32(smem + g.so_a) >> 4, b16 = smem_u32(smem) >> 4;
        const uint32_t hi = 8u | (1u << 14); // SBO 128 bytes, descriptor version, no swizzle
        const uint32_t fmt = KIND == 0 ? 2u : 1u;
        const uint32_t idesc0 = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t) (TC_M >> 4) << 24);
        const uint2* steps = reinterpret_cast<const uint2*>(ct.v);
        const uint4* groups = ct.v + g.co_groups;
        const uint32_t* rowtab = reinterpret_cast<const uint32_t*>(ct.v) + g.co_rows;
        const uint32_t tmem_u = uniform(tmem_base);
        uint32_t slot = (uint32_t) iss_w, a_par = 0; // A ring: this issuer's next slot
        int skip = (int) slot;                                      // staged rows until its next one
        uint32_t stage = 0, b_par = 0;          // filter image stages
        uint32_t first_slot = 0, first_lap = 0; // plane slot that a new plane opens
        uint32_t last_slot = 0;                 // plane slot that completes
        uint32_t phase = 0;
        int kg_have = -1;
#pragma unroll 1
        for (uint32_t unit = blockIdx.x; unit < g.units && ok; unit += gridDim.x)
        {
            const ShUnit u = sh_unit(g, unit);
            if (!g.stream && u.kg != kg_have && u.z_hi > u.z_lo)
            {
                kg_have = u.kg;
                ok = all_lanes(mbar_wait_t<0>(&b_full[0], b_par, abort_flag));
                b_par ^= 1;
            }
            const int nq = (u.nz - g.fs) / g.st_s + 1; // planes opened and closed
            int opened = 0, closed = 0;
#pragma unroll 1
            for (int z = 0; z < u.nz && ok; ++z)
            {
                const bool opens = opened * g.st_s == z && opened < nq, closes = closed * g.st_s + g.fs - 1 == z;
                const bool real = z >= u.z_lo && z < u.z_hi;
                int j_open = opens && first_lap > 0 ? 0 : g.th;
#pragma unroll 1
                for (int grp = 0; grp < g.cgroups && ok; ++grp)
                {
                    uint32_t bset = b16;
                    if (g.stream && real)
                    {
                        ok = all_lanes(mbar_wait_t<0>(&b_full[stage], b_par, abort_flag));
                        bset += stage * (uint32_t) g.b_stage16;
                    }
                    else if (!g.stream)
                        bset += (uint32_t) (grp * g.b_stage16);
                    int j_close = closes && grp + 1 == g.cgroups ? 0 : g.th;
                    int i = real ? u.i_lo + skip : g.rows;
                    const int i_hi = real ? u.i_hi : 0;
                    if (real)
                    {
                        skip -= u.i_hi - u.i_lo;
                        while (skip < 0)
                            skip += SH_ISS;
                    }
#pragma unroll 1
                    for (; i < i_hi && ok; i += SH_ISS)
                    {
                        // what the row does, before waiting for what it needs
                        const uint32_t rt = rowtab[uniform(phase * (uint32_t) g.rows + (uint32_t) i)];
                        const uint32_t g0 = rt & 0xffffu, g1 = g0 + (rt >> 16);
#pragma unroll 1
                        for (; j_open * g.st_r <= i && j_open < g.th && ok; ++j_open)
                            ok = mbar_wait_t<0>(&ev_empty[j_open * g.ns + (int) first_slot], (first_lap - 1) & 1,
                                                abort_flag);
                        ok = all_lanes(ok && mbar_wait_t<0>(&a_full[slot], a_par, abort_flag));
                        if (!ok)
                            break;
                        tc_fence_after();
                        const uint32_t aslot = uniform(a16 + slot * (uint32_t) g.a_slot16), bs = uniform(bset);
#pragma unroll 1
                        for (uint32_t gi = g0; gi < g1; ++gi)
                        {
                            const uint4 gr = groups[gi];
                            const uint32_t d = tmem_u + (gr.x & 0xffffu);
                            const uint32_t idesc = idesc0 | (gr.x >> 16 >> 3 << 17);
                            const uint32_t bb = bs + gr.z;
                            const uint32_t s0 = gr.y & 0xffffu, s1 = s0 + (gr.y >> 16);
#pragma unroll 3
                            for (uint32_t s = s0; s < s1; ++s)
                            {
                                const uint2 st = steps[s];
                                sh_mma<KIND>(d, (uint64_t) hi << 32 | (aslot + st.x), (uint64_t) hi << 32 | (bb + st.y), idesc,
                                             elected);
                            }
                        }
                        if (elected)
                            mma_commit(&a_empty[slot]);
                        slot += SH_ISS;
                        if (slot >= (uint32_t) g.a_slots)
                        {
                            slot -= (uint32_t) g.a_slots;
                            a_par ^= 1;
                        }
                        // blocks whose last row comes before this issuer's next one
#pragma unroll 1
                        for (; j_close * g.st_r + g.fr - 1 < i + sh_reports_ahead(g) && j_close < g.th; ++j_close)
                            if (elected)
                                mma_commit(&ev_full[j_close * g.ns + (int) last_slot]);
                    }
#pragma unroll 1
                    for (; grp == 0 && j_open < g.th && ok; ++j_open)
                        ok = mbar_wait_t<0>(&ev_empty[j_open * g.ns + (int) first_slot], (first_lap - 1) & 1, abort_flag);
                    ok = all_lanes(ok);
#pragma unroll 1
                    for (; j_close < g.th && ok; ++j_close)
                        if (elected)
                            mma_commit(&ev_full[j_close * g.ns + (int) last_slot]);
                    if (g.stream && real)
                    {
                        if (elected)
                            mma_commit(&b_empty[stage]);
                        if (++stage == 2)
                        {
                            stage = 0;
                            b_par ^= 1;
                        }
                    }
                }
                if (opens)
                {
                    ++opened;
                    if (++first_slot == (uint32_t) g.ns)
                    {
                        first_slot = 0;
                        ++first_lap;
                    }
                }
                if (closes)
                {
                    ++closed;
                    if (++last_slot == (uint32_t) g.ns)
                        last_slot = 0;
                }
                if (++phase == (uint32_t) g.nph)
                    phase = 0;
            }
            // the next unit starts at its first plane's phase
            phase = first_slot * (uint32_t) g.st_s;
            if (!g.stream && g.kgroups > 1)
            {
                uint32_t nx = unit + gridDim.x;
                int kg_next = kg_have;
#pragma unroll 1
                for (; nx < g.units; nx += gridDim.x)
                {
                    const ShUnit t = sh_unit(g, nx);
                    if (t.z_hi > t.z_lo)
                    {
                        kg_next = t.kg;
                        break;
                    }
                }
                if (kg_next != kg_have && kg_have >= 0 && elected)
                    mma_commit(&b_empty[0]);
            }
        }
        __syncwarp();
    }
    else if (lane == 0)
    {
        // ------------------------------------------------------------------
        // filter-image loader: the whole image when the filter group changes,
        // or one (plane, channel group) set at a time
        // ------------------------------------------------------------------
        const uint32_t b0 = smem_u32(smem);
        auto load = [&](uint32_t dst, const uint4* src, uint32_t n16, uint64_t* bar) {
            mbar_expect_tx(bar, n16 * 16u);
#pragma unroll 1
            for (uint32_t o = 0; o < n16; o += 2048)
                bulk_load(dst + o * 16u, src + o, (n16 - o < 2048u ? n16 - o : 2048u) * 16u, bar);
        };
        const uint32_t total16 = sets[g.nph].x; // all sets of one (filter group, channel group)
        if (!g.stream)
        {
            int kg_have = -1;
            uint32_t uses = 0;
#pragma unroll 1
            for (uint32_t unit = blockIdx.x; unit < g.units && ok; unit += gridDim.x)
            {
                const ShUnit u = sh_unit(g, unit);
                if (u.kg == kg_have || u.z_hi <= u.z_lo)
                    continue;
                kg_have = u.kg;
                if (uses > 0)
                    ok = mbar_wait(&b_empty[0], (uses - 1) & 1, abort_flag);
                if (!ok)
                    break;
                ++uses;
                load(b0, bimg + (size_t) u.kg * g.cgroups * total16, (uint32_t) g.cgroups * total16, &b_full[0]);
            }
        }
        else
        {
            uint32_t stage = 0, lap = 0;
            uint32_t phase0 = 0;
#pragma unroll 1
            for (uint32_t unit = blockIdx.x; unit < g.units && ok; unit += gridDim.x)
            {
                const ShUnit u = sh_unit(g, unit);
#pragma unroll 1
                for (int z = u.z_lo; z < u.z_hi && ok; ++z)
                {
                    const uint32_t phase = (phase0 + (uint32_t) z) % (uint32_t) g.nph;
#pragma unroll 1
                    for (int grp = 0; grp < g.cgroups && ok; ++grp)
                    {
                        if (lap > 0)
                            ok = mbar_wait(&b_empty[stage], (lap - 1) & 1, abort_flag);
                        if (!ok)
                            break;
                        load(b0 + stage * (uint32_t) g.b_stage16 * 16u,
                             bimg + ((size_t) u.kg * g.cgroups + grp) * total16 + sets[phase].x, sets[phase].y,
                             &b_full[stage]);
                        if (++stage == 2)
                        {
                            stage = 0;
                            ++lap;
                        }
                    }
                }
                const int nq = (u.nz - g.fs) / g.st_s + 1;
                phase0 = (phase0 + (uint32_t) (nq * g.st_s)) % (uint32_t) g.nph;
            }
        }
    }

    if (!ok && lane == 0)
        atomicExch(status, 1);
    // Every role leaves its loop after a bounded time (all waits are bounded
    // and watch the abort flag), so the block-wide barrier is always reached.
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TC_TMEM_COLS)
                     : "memory");
    // (in the one-pass variants the call would cost the converters registers: a kernel of its own)
    if (PARTS == 1)
    {
        if (abort_flag[1] != 0 && tid == 0)
            *ex.out_flag = ex.call;
    }
    else if ((abort_flag[1] != 0 || *ex.w_flag == ex.call) && beta == 0.f)
        sh_repair<STATS>(g, ex, y, stat_part);
}

// sh_repair behind a one-pass kernel, with that kernel's grid.
template <bool STATS>
__global__ void __launch_bounds__(SH_THREADS)
    sh_repair_kernel(const __grid_constant__ ShGeom g, const __grid_constant__ ShExact ex, float* y, float* stat_part)
{
    wait_for_previous_kernel(y);
    if (*ex.out_flag == ex.call || *ex.w_flag == ex.call)
        sh_repair<STATS>(g, ex, y, stat_part);
}

} // namespace dcb
