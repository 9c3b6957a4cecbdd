// Pooling on a halo-extended shard: stands in for cudnnPoolingForward /
// cudnnPoolingBackward behind GPUDNNBackend::pooling_forward / _backward as
// Pooling<BackendDNNLib, T> calls them
// (legacy/include/distconv/dnn_backend/pooling.hpp:212-283).
//
// Both passes are gathers (one thread per result cell, W fastest so that a
// warp reads and writes consecutive cells) and so are reproducible:
//
//   forward   y[o] = alpha * pool(window of o) + beta * y[o]
//   backward  dx[i] = alpha * sum over the windows o that contain i of
//                         MAX:  dy[o] if i is the first cell of o's window (scan
//                               order D, H, W) that holds the maximum, else 0
//                         AVG:  dy[o] / count(o)
//                     + beta * dx[i]
//
// Cells outside the x window are padding: ignored by MAX and by the
// count of AVERAGE_NO_PAD, zeros that count for AVERAGE.  Where a dimension is
// partitioned the caller passes pad 0 and a window that includes the halo
// cells, and the backward pass writes the halo cells of dx too; the reverse
// halo exchange with SUM then adds them to their owners
// (pooling.hpp:281, :450-467).  The halo cells of a rank at the boundary of
// the global tensor stand for padding (pooling.hpp:189-194); the reference
// hands them to cuDNN as zero data, which changes MAX and AVERAGE_NO_PAD
// against the unpartitioned result.  Here the descriptor says how many leading
// / trailing cells of the window lie outside the global tensor and those are
// padding like any other, so P ranks give what one rank gives.
//
// HBM-bound: algorithmic bytes are 4 * (|x| + |y|) forward and
// 4 * (|x| + |y| + |dy| + |dx|) backward; the window re-reads hit L1 / L2.
#include "common.cuh"
#include "dcb.h"

#include <cfloat>
#include <type_traits>

namespace dcb
{
namespace
{

struct PoolGeom
{
    int n, c;
    int in[3], out[3], win[3], pad[3], stride[3];
    int lo[3], hi[3]; // real cells of the x window along each axis: [lo, hi)
    long long xs_n, xs_c, xs[3];
    long long ys_n, ys_c, ys[3];
    int mode;
};

constexpr int POOL_THREADS = 256;

// Cells along axis i that output o's average is over.
__device__ __forceinline__ int pool_extent(const PoolGeom& g, int i, int o)
{
    if (g.mode == DCB_POOL_AVERAGE)
        return g.win[i];
    const int lo = max(g.lo[i], o * g.stride[i] - g.pad[i]), hi = min(g.hi[i], o * g.stride[i] - g.pad[i] + g.win[i]);
    return max(0, hi - lo);
}

__device__ __forceinline__ float pool_count(const PoolGeom& g, int od, int oh, int ow)
{
    if (g.mode == DCB_POOL_AVERAGE)
        return (float) (g.win[0] * g.win[1] * g.win[2]);
    return (float) (pool_extent(g, 0, od) * pool_extent(g, 1, oh) * pool_extent(g, 2, ow));
}

// row = plane * extent + line, with the 32-bit division when the row count allows it
// (the 64-bit one is a subroutine of a hundred instructions)
__device__ __forceinline__ void pool_split_row(long long row, long long rows, int extent, int* plane, int* line)
{
    if (rows <= 0x7fffffffll)
    {
        const unsigned r = (unsigned) row, e = (unsigned) extent;
        *plane = (int) (r / e);
        *line = (int) (r - (r / e) * e);
    }
    else
    {
        *plane = (int) (row / extent);
        *line = (int) (row % extent);
    }
}

// Forward: one thread per output cell, the window scanned in D, H, W order.
// `argmax`, if given, receives the tap index kd * fh * fw + kh * fw + kw of the
// first maximum (dense [n][c][od][oh][ow]); y may then be null.
constexpr int POOL_TW = POOL_THREADS;

__global__ void __launch_bounds__(POOL_THREADS)
    pool_fwd_kernel(PoolGeom g, float alpha, float beta, const float* __restrict__ x, float* y,
                    unsigned char* __restrict__ argmax, int tw_log2, long long rows)
{
    const int w0_ = g.win[0], w1_ = g.win[1], w2_ = g.win[2], s0_ = g.stride[0], s1_ = g.stride[1], s2_ = g.stride[2];
    // a block is 256 >> tw_log2 output rows of (1 << tw_log2) cells: short rows (128
    // outputs of a 256-cell input row) would otherwise leave half the block idle
    const int ow = (blockIdx.y << tw_log2) + (threadIdx.x & ((1 << tw_log2) - 1));
    const long long row = (long long) blockIdx.x * (POOL_THREADS >> tw_log2) + (threadIdx.x >> tw_log2);
    if (ow >= g.out[2] || row >= rows)
        return;
    const int oh = (int) (row % g.out[1]), od = (int) (row / g.out[1]);
    const int c = blockIdx.z % g.c, n = blockIdx.z / g.c;
    const float* xp = x + (size_t) n * g.xs_n + (size_t) c * g.xs_c;
    const int d0 = od * s0_ - g.pad[0], h0 = oh * s1_ - g.pad[1], w0 = ow * s2_ - g.pad[2];
    const int kw_lo = max(0, g.lo[2] - w0), kw_hi = min(w2_, g.hi[2] - w0);
    float m = -FLT_MAX, s = 0.f;
    int best = -1;
    for (int kd = 0; kd < w0_; ++kd)
    {
        const int id = d0 + kd;
        if (id < g.lo[0] || id >= g.hi[0])
            continue;
        for (int kh = 0; kh < w1_; ++kh)
        {
            const int ih = h0 + kh;
            if (ih < g.lo[1] || ih >= g.hi[1])
                continue;
            const float* row = xp + (size_t) id * g.xs[0] + (size_t) ih * g.xs[1] + w0;
            const int tap0 = (kd * w1_ + kh) * w2_;
            for (int kw = 0; kw < w2_; ++kw)
            {
                if (kw < kw_lo || kw >= kw_hi)
                    continue;
                const float v = __ldg(row + kw);
                s += v;
                if (best < 0 || v > m)
                {
                    m = v;
                    best = tap0 + kw;
                }
            }
        }
    }
    if (argmax)
    {
        argmax[((((size_t) n * g.c + c) * g.out[0] + od) * g.out[1] + oh) * g.out[2] + ow] = (unsigned char) best;
        if (!y)
            return;
    }
    const float r = g.mode == DCB_POOL_MAX ? m : s / fmaxf(pool_count(g, od, oh, ow), 1.f);
    float* yp = y + (size_t) n * g.ys_n + (size_t) c * g.ys_c + (size_t) od * g.ys[0] + (size_t) oh * g.ys[1] + ow;
    *yp = beta != 0.f ? alpha * r + beta * *yp : alpha * r;
}

// The same for the common windows, O neighbouring outputs a thread (launch_pool_general): a window
// row's cells are loaded once for all of them and the addresses worked out once.  Same scan order,
// same bits.  Bound by what a thread does per cell.  (us, an output a thread with a check per cell
// before: 8 x 128^3, 3 / 1, averages 309 -> 124; 16 x 64 x 100 x 90, maxima, 2 / 2 18.5 -> 11.8, 3 / 1 177 -> 133;
// 4 x 16^3, maxima, 3 / 1 4.2 -> 3.9.)
template <int WD, int W, int S, bool MAXP, int O>
__global__ void __launch_bounds__(POOL_THREADS)
    pool_fwd_cells_kernel(PoolGeom g, float alpha, float beta, const float* __restrict__ x, float* y,
                          unsigned char* __restrict__ argmax, int tw_log2, long long rows)
{
    constexpr int SD = WD == 1 ? 1 : S, NC = (O - 1) * S + W; // cells behind O outputs
    const int ow0 = ((blockIdx.y << tw_log2) + (threadIdx.x & ((1 << tw_log2) - 1))) * O;
    const long long row = (long long) blockIdx.x * (POOL_THREADS >> tw_log2) + (threadIdx.x >> tw_log2);
    if (ow0 >= g.out[2] || row >= rows)
        return;
    int od, oh;
    pool_split_row(row, rows, g.out[1], &od, &oh);
    const int c = blockIdx.z % g.c, n = blockIdx.z / g.c;
    const int d0 = od * SD - g.pad[0], h0 = oh * S - g.pad[1], w0 = ow0 * S - g.pad[2];
    const float* xp = x + (size_t) n * g.xs_n + (size_t) c * g.xs_c + (long long) d0 * g.xs[0] + (long long) h0 * g.xs[1] + w0;
    const bool all = w0 >= g.lo[2] && w0 + NC <= g.hi[2]; // every cell exists
    float r[O];
    int best[O];
    bool first = true;
#pragma unroll
    for (int o = 0; o < O; ++o)
        r[o] = MAXP ? -FLT_MAX : 0.f, best[o] = -1;
#pragma unroll
    for (int kd = 0; kd < WD; ++kd)
    {
        if (d0 + kd < g.lo[0] || d0 + kd >= g.hi[0])
            continue;
        // a plane's rows before the first is looked at: their loads are in flight together
        // (3 / 1, maxima 172 -> 155 us)
        float v[W][NC];
#pragma unroll
        for (int kh = 0; kh < W; ++kh)
        {
            const float* rp = xp + kd * g.xs[0] + kh * g.xs[1];
            const bool row_in = h0 + kh >= g.lo[1] && h0 + kh < g.hi[1];
#pragma unroll
            for (int i = 0; i < NC; ++i)
                v[kh][i] = row_in && (all || (w0 + i >= g.lo[2] && w0 + i < g.hi[2])) ? __ldg(rp + i) : (MAXP ? -INFINITY : 0.f);
        }
#pragma unroll
        for (int kh = 0; kh < W; ++kh)
        {
            if (h0 + kh < g.lo[1] || h0 + kh >= g.hi[1])
                continue;
            if (MAXP && first)
            {
                // the first cell that exists, whatever it holds (a NaN stays the maximum)
                first = false;
#pragma unroll
                for (int o = 0; o < O; ++o)
#pragma unroll
                    for (int kw = W - 1; kw >= 0; --kw)
                        if (all || (w0 + o * S + kw >= g.lo[2] && w0 + o * S + kw < g.hi[2]))
                        {
                            r[o] = v[kh][o * S + kw];
                            best[o] = (kd * W + kh) * W + kw;
                        }
            }
#pragma unroll
            for (int o = 0; o < O; ++o)
#pragma unroll
                for (int kw = 0; kw < W; ++kw)
                {
                    // (cells that do not exist add nothing and are no greater than any)
                    if (!MAXP)
                        r[o] += v[kh][o * S + kw];
                    else if (v[kh][o * S + kw] > r[o])
                    {
                        r[o] = v[kh][o * S + kw];
                        best[o] = (kd * W + kh) * W + kw;
                    }
                }
        }
    }
    const int left = min(O, g.out[2] - ow0);
    if (argmax)
    {
        unsigned char* ap = argmax + ((((size_t) n * g.c + c) * g.out[0] + od) * g.out[1] + oh) * g.out[2] + ow0;
#pragma unroll
        for (int o = 0; o < O; ++o)
            if (o < left)
                ap[o] = (unsigned char) best[o];
        if (!y)
            return;
    }
    float* yp = y + (size_t) n * g.ys_n + (size_t) c * g.ys_c + (size_t) od * g.ys[0] + (size_t) oh * g.ys[1] + ow0;
#pragma unroll
    for (int o = 0; o < O; ++o)
        if (o < left)
        {
            const float q = MAXP ? r[o] : r[o] / fmaxf(pool_count(g, od, oh, ow0 + o), 1.f);
            yp[o] = beta != 0.f ? alpha * q + beta * yp[o] : alpha * q;
        }
}

// Forward for windows of 3 with stride 2 and pad 1 along W (and H; WD = 3 with stride 2
// or 1 with stride 1 along D) on rows that start on 16-byte boundaries: a thread takes
// two neighbouring outputs, i.e. input cells 4t-1 .. 4t+3 of every window row: one
// 16-byte load and the left neighbour's last cell from a shuffle, where the one-output
// kernel issues six scalar loads at every second cell.  Same scan order (D, H, W, first
// maximum wins), same arithmetic.
template <int WD>
__global__ void __launch_bounds__(POOL_THREADS)
    pool_fwd_w3s2_kernel(PoolGeom g, float alpha, float beta, const float* __restrict__ x, float* y,
                         unsigned char* __restrict__ argmax, int tw_log2, long long rows)
{
    const int tq = (blockIdx.y << tw_log2) + (threadIdx.x & ((1 << tw_log2) - 1)); // pair of outputs
    const long long row = (long long) blockIdx.x * (POOL_THREADS >> tw_log2) + (threadIdx.x >> tw_log2);
    const bool live = 2 * tq < g.out[2] && row < rows; // dead lanes still take part in the shuffles
    int oh, od;
    pool_split_row(row, rows, g.out[1], &od, &oh);
    const int c = blockIdx.z % g.c, n = blockIdx.z / g.c;
    const float* xp = x + (size_t) n * g.xs_n + (size_t) c * g.xs_c;
    // offsets inside one (sample, channel) volume fit 32 bits (checked at the launch)
    const int xs0 = (int) g.xs[0], xs1 = (int) g.xs[1];
    const int sd = WD == 1 ? 1 : 2;
    const int d0 = od * sd - g.pad[0], h0 = oh * 2 - g.pad[1];
    const int w4 = 4 * tq; // cells w4 - 1 .. w4 + 3
    float m[2] = {-FLT_MAX, -FLT_MAX}, s[2] = {0.f, 0.f};
    int best[2] = {-1, -1};
    const int lane = threadIdx.x & 31;
    // A warp whose windows all lie inside the real cells (every warp but those at the
    // faces) runs without range checks: tap 0 is then every window's first cell, so the
    // "first cell always becomes the maximum" rule is an assignment there and a plain
    // comparison after it.  Same results as the checked loop below.
    const bool full = live && 2 * tq + 1 < g.out[2] && d0 >= g.lo[0] && d0 + WD <= g.hi[0] && h0 >= g.lo[1]
                      && h0 + 3 <= g.hi[1] && w4 >= g.lo[2] && w4 + 3 < g.hi[2];
    const bool fast = __all_sync(0xffffffffu, full);
    // the first thread of a row: its cell w4 - 1 is the padding, tap 1 its first window's first cell
    const bool ledge = w4 - 1 < g.lo[2];
    if (fast)
    {
        const float* rp0 = xp + (d0 * xs0 + h0 * xs1 + w4);
        const bool want_max = g.mode == DCB_POOL_MAX;
#pragma unroll
        for (int kd = 0; kd < WD; ++kd)
#pragma unroll
            for (int kh = 0; kh < 3; ++kh)
            {
                const float* rp = rp0 + (kd * xs0 + kh * xs1);
                const float4 t = __ldg(reinterpret_cast<const float4*>(rp));
                float prev = __shfl_up_sync(0xffffffffu, t.w, 1);
                if (lane == 0 && !ledge)
                    prev = __ldg(rp - 1);
                const float v[5] = {prev, t.x, t.y, t.z, t.w};
                const int tap0 = (kd * 3 + kh) * 3;
                if (want_max)
                {
#pragma unroll
                    for (int o = 0; o < 2; ++o)
#pragma unroll
                        for (int kw = 0; kw < 3; ++kw)
                        {
                            const float val = v[2 * o + kw];
                            const bool row0 = kd == 0 && kh == 0;
                            bool take;
                            if (o == 0 && kw == 0)
                                take = !ledge && (row0 || val > m[o]);
                            else if (o == 0 && kw == 1 && row0)
                                take = ledge || val > m[o];
                            else
                                take = (row0 && kw == 0) || val > m[o];
                            if (take)
                            {
                                m[o] = val;
                                best[o] = tap0 + kw;
                            }
                        }
                }
                else
                {
                    s[0] += ledge ? 0.f : v[0];
                    s[0] += v[1];
                    s[0] += v[2];
#pragma unroll
                    for (int kw = 0; kw < 3; ++kw)
                        s[1] += v[2 + kw];
                }
            }
    }
#pragma unroll
    for (int kd = 0; kd < WD && !fast; ++kd)
    {
        const int id = d0 + kd;
        const bool dok = live && id >= g.lo[0] && id < g.hi[0];
#pragma unroll
        for (int kh = 0; kh < 3; ++kh)
        {
            const int ih = h0 + kh;
            const bool rok = dok && ih >= g.lo[1] && ih < g.hi[1];
            float q[4] = {0.f, 0.f, 0.f, 0.f};
            if (rok)
            {
                const float* rp = xp + (id * xs0 + ih * xs1 + w4);
                if (w4 + 3 < g.hi[2])
                {
                    const float4 t = __ldg(reinterpret_cast<const float4*>(rp));
                    q[0] = t.x;
                    q[1] = t.y;
                    q[2] = t.z;
                    q[3] = t.w;
                }
                else
                {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (w4 + e < g.hi[2])
                            q[e] = __ldg(rp + e);
                }
            }
            // cell w4 - 1: the left neighbour's q[3] (same output row: a tile is 32 lanes or more)
            float prev = __shfl_up_sync(0xffffffffu, q[3], 1);
            if (lane == 0 && rok && w4 - 1 >= g.lo[2])
                prev = __ldg(xp + (id * xs0 + ih * xs1 + w4 - 1));
            if (!rok)
                continue;
            const float v[5] = {prev, q[0], q[1], q[2], q[3]};
            const int tap0 = (kd * 3 + kh) * 3;
#pragma unroll
            for (int o = 0; o < 2; ++o)
#pragma unroll
                for (int kw = 0; kw < 3; ++kw)
                {
                    const int cell = w4 - 1 + 2 * o + kw;
                    if (cell < g.lo[2] || cell >= g.hi[2])
                        continue;
                    const float val = v[2 * o + kw];
                    s[o] += val;
                    if (best[o] < 0 || val > m[o])
                    {
                        m[o] = val;
                        best[o] = tap0 + kw;
                    }
                }
        }
    }
    if (!live)
        return;
#pragma unroll
    for (int o = 0; o < 2; ++o)
    {
        const int ow = 2 * tq + o;
        if (ow >= g.out[2])
            continue;
        if (argmax)
            argmax[((size_t) n * g.c + c) * ((size_t) g.out[0] * g.out[1] * g.out[2]) + ((od * g.out[1] + oh) * g.out[2] + ow)] =
                (unsigned char) best[o];
        if (!y)
            continue;
        const float r = g.mode == DCB_POOL_MAX ? m[o] : s[o] / fmaxf(pool_count(g, od, oh, ow), 1.f);
        float* yp =
            y + (size_t) n * g.ys_n + (size_t) c * g.ys_c + (od * (int) g.ys[0] + oh * (int) g.ys[1] + ow);
        *yp = beta != 0.f ? alpha * r + beta * *yp : alpha * r;
    }
}

// The same for windows of 3 with stride 2 along D too, the usual down-sampling of a
// volume: a thread walks along D with its pair of outputs.  Window od covers planes
// 2 od - pad .. + 2, so every second plane belongs to two windows: its maximum over the
// thread's 3 x 5 cells (position, and first cell for the rule below) is carried over.  A
// plane is then read and scanned once instead of 1.5 times; what is left is the overlap
// of neighbouring output rows along H, which L1 has.
// The scan's rule is "the window's first cell becomes the maximum, a later cell if it
// is larger": a first cell that is not a number stays the maximum.  A plane's own
// maximum is therefore taken over numbers only (start -inf), and the first cell is
// looked at again where the plane opens a window.  Same results, bit for bit.
// 16 x 256^3 floats, maximum: 312 -> 221 us forward, 312 -> 246 us for the indices of the
// backward pass (184 and 170 us at the rate of a copy).  Bound by latency: four blocks an
// SM (64 registers; with 80 and three blocks the index pass takes 264 us), six 16-byte
// loads in flight per thread (three, with the range checks between them: 301 and 379 us).
struct PoolPlane
{
    float m[2], f[2]; // maximum (or sum) and first cell, per output of the pair
    int t[2];         // tap kh * 3 + kw of the maximum
};

template <bool MAXP, bool IDX>
__global__ void __launch_bounds__(POOL_THREADS, 4)
    pool_fwd_march_kernel(PoolGeom g, float alpha, float beta, const float* __restrict__ x, float* y,
                          unsigned char* __restrict__ argmax, int tw_log2, long long rows, int seg)
{
    const int tq = (blockIdx.y << tw_log2) + (threadIdx.x & ((1 << tw_log2) - 1)); // pair of outputs
    const long long row = (long long) blockIdx.x * (POOL_THREADS >> tw_log2) + (threadIdx.x >> tw_log2);
    if (row >= rows) // a warp never spans two rows: the whole warp leaves
        return;
    int s, oh;
    pool_split_row(row, rows, g.out[1], &s, &oh);
    const int c = blockIdx.z % g.c, n = blockIdx.z / g.c, lane = threadIdx.x & 31;
    const bool live = 2 * tq < g.out[2], both = 2 * tq + 1 < g.out[2]; // dead lanes still take part in the shuffles
    const int xs0 = (int) g.xs[0], xs1 = (int) g.xs[1];
    const int h0 = oh * 2 - g.pad[1], w4 = 4 * tq; // cells w4 - 1 .. w4 + 3
    const float* xp = x + (size_t) n * g.xs_n + (size_t) c * g.xs_c + (h0 * xs1 + w4);
    const bool ledge = tq == 0, whole = w4 + 3 < g.in[2];
    const float none = MAXP ? __int_as_float(0xff800000) : 0.f; // of a cell that does not exist
    const bool any_row = max(h0, g.lo[1]) < min(h0 + 3, g.hi[1]);

    // a plane's cells; FAST: all exist, no branches, so that all loads of a step are in flight together
    auto load = [&](int id, float (&v)[3][5], auto fast) {
#pragma unroll
        for (int kh = 0; kh < 3; ++kh)
        {
            const float* rp = xp + (id * xs0 + kh * xs1);
            if (fast.value)
            {
                const float4 q = __ldg(reinterpret_cast<const float4*>(rp));
                v[kh][1] = q.x, v[kh][2] = q.y, v[kh][3] = q.z, v[kh][4] = q.w;
                v[kh][0] = none;
                if (lane == 0 && !ledge)
                    v[kh][0] = __ldg(rp - 1);
                continue;
            }
            v[kh][0] = v[kh][1] = v[kh][2] = v[kh][3] = v[kh][4] = none;
            if (h0 + kh >= g.lo[1] && h0 + kh < g.hi[1]) // the same for the whole warp
            {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (w4 + e < g.in[2])
                        v[kh][1 + e] = __ldg(rp + e);
                if (lane == 0 && live && !ledge)
                    v[kh][0] = __ldg(rp - 1);
            }
        }
    };
    auto scan = [&](float (&v)[3][5], PoolPlane& p, auto fast) {
        p.m[0] = p.m[1] = none;
        p.f[0] = p.f[1] = none;
        p.t[0] = p.t[1] = 0;
        bool seen = false;
#pragma unroll
        for (int kh = 0; kh < 3; ++kh)
        {
            // cell w4 - 1 is the left neighbour's last one
            const float left = __shfl_up_sync(0xffffffffu, v[kh][4], 1);
            if (lane != 0)
                v[kh][0] = left;
            if (!fast.value && (h0 + kh < g.lo[1] || h0 + kh >= g.hi[1]))
                continue;
            if (MAXP && !seen)
            {
                seen = true;
                p.f[0] = ledge ? v[kh][1] : v[kh][0];
                p.f[1] = v[kh][2];
                p.t[0] = kh * 3 + (ledge ? 1 : 0);
                p.t[1] = kh * 3;
            }
#pragma unroll
            for (int o = 0; o < 2; ++o)
#pragma unroll
                for (int kw = 0; kw < 3; ++kw)
                {
                    const float val = v[kh][2 * o + kw];
                    if (!MAXP)
                        p.m[o] += val;
                    else if (val > p.m[o])
                    {
                        p.m[o] = val;
                        if (IDX)
                            p.t[o] = kh * 3 + kw;
                    }
                }
        }
    };

    const int od0 = s * seg, od1 = min(od0 + seg, g.out[0]);
    PoolPlane carry, mid, next;
    int id = 2 * od0 - g.pad[0];
    const std::false_type checked{};
    auto scan_checked = [&](int plane, PoolPlane& p) {
        float v[3][5];
        if (plane >= g.lo[0] && plane < g.hi[0]) // the same for the whole warp
            load(plane, v, checked), scan(v, p, checked);
        else
            p = {{none, none}, {none, none}, {0, 0}};
    };
    const bool inside = __all_sync(0xffffffffu, live && whole) && h0 >= g.lo[1] && h0 + 3 <= g.hi[1];
    if (inside && id >= g.lo[0] && id < g.hi[0])
    {
        float v[3][5];
        load(id, v, std::true_type{});
        scan(v, carry, std::true_type{});
    }
    else
        scan_checked(id, carry);
    // every cell that the walk has yet to read exists
    const bool fast = inside && id + 1 >= g.lo[0] && id + 2 * (od1 - od0) < g.hi[0];
    for (int od = od0; od < od1; ++od, id += 2)
    {
        if (fast)
        {
            float v[3][5], w[3][5];
            load(id + 1, v, std::true_type{});
            load(id + 2, w, std::true_type{});
            scan(v, mid, std::true_type{});
            scan(w, next, std::true_type{});
        }
        else
        {
            scan_checked(id + 1, mid);
            scan_checked(id + 2, next);
        }
        float r[2];
        int b[2];
#pragma unroll
        for (int o = 0; o < 2; ++o)
        {
            if (!MAXP)
            {
                r[o] = (carry.m[o] + mid.m[o] + next.m[o]) / fmaxf(pool_count(g, od, oh, 2 * tq + o), 1.f);
                continue;
            }
            bool open = false; // the window has had its first cell
            r[o] = -FLT_MAX;
            b[o] = -1;
            const PoolPlane* const pl[3] = {&carry, &mid, &next};
#pragma unroll
            for (int kd = 0; kd < 3; ++kd)
            {
                if (!any_row || id + kd < g.lo[0] || id + kd >= g.hi[0])
                    continue;
                if (!open)
                {
                    const bool nan = !(pl[kd]->f[o] == pl[kd]->f[o]);
                    r[o] = nan ? pl[kd]->f[o] : pl[kd]->m[o];
                    // the first valid tap: without numbers above -inf t still says where that is
                    b[o] = kd * 9 + pl[kd]->t[o];
                    if (IDX && nan)
                    {
                        const int first = max(0, g.lo[1] - h0) * 3 + (o == 0 && ledge ? 1 : 0);
                        b[o] = kd * 9 + first;
                    }
                    open = true;
                }
                else if (pl[kd]->m[o] > r[o])
                {
                    r[o] = pl[kd]->m[o];
                    b[o] = kd * 9 + pl[kd]->t[o];
                }
            }
        }
        carry = next;
        if (!live)
            continue;
        if (IDX)
        {
            unsigned char* ap = argmax + ((size_t) n * g.c + c) * ((size_t) g.out[0] * g.out[1] * g.out[2])
                                + ((od * g.out[1] + oh) * g.out[2] + 2 * tq);
            if (both && (reinterpret_cast<uintptr_t>(ap) & 1) == 0)
                *reinterpret_cast<uchar2*>(ap) = make_uchar2((unsigned char) b[0], (unsigned char) b[1]);
            else
            {
                ap[0] = (unsigned char) b[0];
                if (both)
                    ap[1] = (unsigned char) b[1];
            }
        }
        if (!IDX || y)
        {
            float* yp = y + (size_t) n * g.ys_n + (size_t) c * g.ys_c + (od * (int) g.ys[0] + oh * (int) g.ys[1] + 2 * tq);
            if (both && (reinterpret_cast<uintptr_t>(yp) & 7) == 0)
            {
                float2 out = make_float2(alpha * r[0], alpha * r[1]);
                if (beta != 0.f)
                {
                    const float2 old = *reinterpret_cast<const float2*>(yp);
                    out.x += beta * old.x;
                    out.y += beta * old.y;
                }
                *reinterpret_cast<float2*>(yp) = out;
            }
            else
            {
                yp[0] = beta != 0.f ? alpha * r[0] + beta * yp[0] : alpha * r[0];
                if (both)
                    yp[1] = beta != 0.f ? alpha * r[1] + beta * yp[1] : alpha * r[1];
            }
        }
    }
}

// The outputs whose window holds input coordinate i: o*stride - pad <= i < o*stride - pad + win.
__device__ __forceinline__ void pool_cover(int i, int stride, int pad, int win, int nout, int* lo, int* hi)
{
    const int t = i + pad;
    const int l = t - win + 1;
    int lq, hq; // ceil(l / stride) for l > 0, floor(t / stride); strides 1 and 2 without a division
    if (stride == 1)
    {
        lq = l;
        hq = t;
    }
    else if (stride == 2)
    {
        lq = (l + 1) >> 1;
        hq = t >> 1;
    }
    else
    {
        lq = (l + stride - 1) / stride;
        hq = t / stride;
    }
    *lo = l <= 0 ? 0 : lq;
    *hi = min(hq, nout - 1);
}

// Maximum, backward, without a workspace: a thread per input cell looks at the windows that hold it
// and scans those whose maximum it equals.
template <int WD, int W, int S>
__global__ void __launch_bounds__(POOL_THREADS)
    pool_bwd_kernel(PoolGeom g, float alpha, float beta, const float* __restrict__ y, const float* __restrict__ dy,
                    const float* __restrict__ x, float* dx)
{
    // window / stride as compile-time constants where the launch found a match
    // (unrolled loops, shifts for the divisions); 0 = read them from the geometry
    const int w0_ = WD ? WD : g.win[0], w1_ = W ? W : g.win[1], w2_ = W ? W : g.win[2];
    const int s0_ = S ? (WD == 1 ? 1 : S) : g.stride[0], s1_ = S ? S : g.stride[1], s2_ = S ? S : g.stride[2];
    const int iw = blockIdx.y * POOL_THREADS + threadIdx.x;
    if (iw >= g.in[2])
        return;
    const int ih = blockIdx.x % g.in[1], id = blockIdx.x / g.in[1];
    const int c = blockIdx.z % g.c, n = blockIdx.z / g.c;
    const size_t xoff = (size_t) n * g.xs_n + (size_t) c * g.xs_c;
    const size_t yoff = (size_t) n * g.ys_n + (size_t) c * g.ys_c;
    const size_t me = xoff + (size_t) id * g.xs[0] + (size_t) ih * g.xs[1] + iw;
    int dlo, dhi, hlo, hhi, wlo, whi;
    pool_cover(id, s0_, g.pad[0], w0_, g.out[0], &dlo, &dhi);
    pool_cover(ih, s1_, g.pad[1], w1_, g.out[1], &hlo, &hhi);
    pool_cover(iw, s2_, g.pad[2], w2_, g.out[2], &wlo, &whi);
    const float xv = __ldg(x + me);
    float acc = 0.f;
    // a cell outside the global tensor is padding: no window gives it anything
    const bool real = id >= g.lo[0] && id < g.hi[0] && ih >= g.lo[1] && ih < g.hi[1] && iw >= g.lo[2] && iw < g.hi[2];
    if (!real)
        dhi = dlo - 1;
    for (int od = dlo; od <= dhi; ++od)
        for (int oh = hlo; oh <= hhi; ++oh)
            for (int ow = wlo; ow <= whi; ++ow)
            {
                const size_t o = yoff + (size_t) od * g.ys[0] + (size_t) oh * g.ys[1] + ow;
                if (__ldg(y + o) != xv)
                    continue;
                // the maximum goes to the first cell that holds it: is one before me?
                bool first = true;
                const int d0 = od * s0_ - g.pad[0], h0 = oh * s1_ - g.pad[1],
                          w0 = ow * s2_ - g.pad[2];
                for (int jd = max(d0, g.lo[0]); jd <= id && first; ++jd)
                    for (int jh = max(h0, g.lo[1]); jh < min(h0 + w1_, g.hi[1]) && first; ++jh)
                    {
                        if (jd == id && jh > ih)
                            break;
                        const float* row = x + xoff + (size_t) jd * g.xs[0] + (size_t) jh * g.xs[1];
                        const int wend = (jd == id && jh == ih) ? iw : min(w0 + w2_, g.hi[2]);
                        for (int jw = max(w0, g.lo[2]); jw < wend; ++jw)
                            if (__ldg(row + jw) == xv)
                            {
                                first = false;
                                break;
                            }
                    }
                if (first)
                    acc += __ldg(dy + o);
            }
    dx[me] = beta != 0.f ? alpha * acc + beta * dx[me] : alpha * acc;
}

// Backward for any window: averages, and maxima by the index workspace.  A thread owns E
// consecutive cells of an input row and walks the windows that hold the row, each gradient (and
// index byte, or quotient) once for all of them.  Short rows share a block; with UNIFORM a block is
// one row, and what depends on the row is worked out once for all its threads (rows of more than 128
// cells; us, rows sharing a block / like this: maxima, 3 / 2, 32 x 27 x 120 x 181 218 / 191, 8 x 112 x 59 x
// 157 112 / 101, averages 75.7 / 67.4; the loops of a general window gain nothing).  Bound by
// instruction issue: what a thread does per window is what counts (us, a cell a thread for averages
// and one row a block before: 2 x 16 x 100 x 96 x 128, 3 / 2, averages 644 -> 217; 8 x 128^3, 3 / 1,
// averages 940 -> 411; 16 x 64 x 100 x 90, 2 / 2, maxima 68 -> 54; 4 x 30 x 30 x 31, 3 / 1, 28.5 -> 9).
template <int WD, int W, int S, bool MAXP, int E, bool UNIFORM>
__global__ void __launch_bounds__(POOL_THREADS)
    pool_bwd_cells_kernel(PoolGeom g, float alpha, float beta, const float* __restrict__ dy, float* dx,
                          const unsigned char* __restrict__ argmax, int tw_log2, long long rows)
{
    const int w0_ = WD ? WD : g.win[0], w1_ = W ? W : g.win[1], w2_ = W ? W : g.win[2];
    const int s0_ = S ? (WD == 1 ? 1 : S) : g.stride[0], s1_ = S ? S : g.stride[1], s2_ = S ? S : g.stride[2];
    const int iw0 = ((blockIdx.y << tw_log2) + (UNIFORM ? threadIdx.x : threadIdx.x & ((1 << tw_log2) - 1))) * E;
    const long long row = UNIFORM ? blockIdx.x : (long long) blockIdx.x * (POOL_THREADS >> tw_log2) + (threadIdx.x >> tw_log2);
    if (iw0 >= g.in[2] || row >= rows)
        return;
    int id, ih;
    pool_split_row(row, rows, g.in[1], &id, &ih);
    const int c = blockIdx.z % g.c, n = blockIdx.z / g.c;
    float acc[E] = {};
    int dlo, dhi, hlo, hhi;
    pool_cover(id, s0_, g.pad[0], w0_, g.out[0], &dlo, &dhi);
    pool_cover(ih, s1_, g.pad[1], w1_, g.out[1], &hlo, &hhi);
    if (id < g.lo[0] || id >= g.hi[0] || ih < g.lo[1] || ih >= g.hi[1])
        dhi = dlo - 1; // a row outside the global tensor is padding
    int wlo[E], whi[E], first = g.out[2], last = -1; // windows of each cell, of all
#pragma unroll
    for (int e = 0; e < E; ++e)
    {
        pool_cover(iw0 + e, s2_, g.pad[2], w2_, g.out[2], &wlo[e], &whi[e]);
        if (iw0 + e < g.lo[2] || iw0 + e >= g.hi[2] || iw0 + e >= g.in[2])
            whi[e] = wlo[e] - 1;
        if (whi[e] >= wlo[e])
            first = min(first, wlo[e]), last = max(last, whi[e]);
    }
    // stride 1: the loads of all windows along W go out together (maxima of 16 x 64 x 100 x 90
    // 365 -> 325 us, averages of 8 x 128^3 488 -> 411; with stride 2 there are two or three, and
    // a fixed number of them costs more: averages of 2 x 16 x 100 x 96 x 128 231 -> 320)
    constexpr int M = S == 1 ? W + E - 1 : 1;
    const size_t plane = ((size_t) n * g.c + c) * g.out[0];
    const float* dyp = dy + (size_t) n * g.ys_n + (size_t) c * g.ys_c;
    for (int od = dlo; od <= dhi; ++od)
        for (int oh = hlo; oh <= hhi; ++oh)
        {
            const unsigned char* arow = argmax + ((plane + od) * g.out[1] + oh) * g.out[2];
            const float* dyrow = dyp + (size_t) od * g.ys[0] + (size_t) oh * g.ys[1];
            const int tap0 = ((id - (od * s0_ - g.pad[0])) * w1_ + (ih - (oh * s1_ - g.pad[1]))) * w2_ + g.pad[2] + iw0;
            // (windows of 2 with stride 2: one window a cell, nothing to share.  us like that / so: 16 x 256^3
            // 998 / 928, 64 x 16 x 200 x 130 196 / 173, 64 x 100 x 90 x 16 34 / 33, 16 x 64 x 100 x 90 48 / 50)
            const int cells = MAXP || W == 2 ? 0 : pool_extent(g, 0, od) * pool_extent(g, 1, oh);
            for (int ow0 = first; ow0 <= last; ow0 += M)
            {
                float d[M];
                int tap[M]; // the cell that the maximum is, of the four
#pragma unroll
                for (int k = 0; k < M; ++k)
                {
                    const int ow = ow0 + k;
                    d[k] = ow <= last ? __ldg(dyrow + ow) : 0.f;
                    tap[k] = MAXP && ow <= last ? (int) __ldg(arow + ow) - (tap0 - ow * s2_) : -1;
                }
#pragma unroll
                for (int k = 0; k < M; ++k)
                {
                    const int ow = ow0 + k;
                    if (!MAXP)
                        d[k] /= fmaxf(W == 2 ? pool_count(g, od, oh, ow) : (float) (cells * pool_extent(g, 2, ow)), 1.f);
#pragma unroll
                    for (int e = 0; e < E; ++e)
                        if (ow >= wlo[e] && ow <= whi[e] && (!MAXP || tap[k] == e))
                            acc[e] += d[k];
                }
            }
        }
    float* xp = dx + (size_t) n * g.xs_n + (size_t) c * g.xs_c + (size_t) id * g.xs[0] + (size_t) ih * g.xs[1] + iw0;
    if (E == 4 && iw0 + 4 <= g.in[2] && (reinterpret_cast<uintptr_t>(xp) & 15) == 0)
    {
        float4 o = make_float4(alpha * acc[0], alpha * acc[E > 1 ? 1 : 0], alpha * acc[E > 2 ? 2 : 0], alpha * acc[E > 3 ? 3 : 0]);
        if (beta != 0.f)
        {
            const float4 old = *reinterpret_cast<const float4*>(xp);
            o.x += beta * old.x;
            o.y += beta * old.y;
            o.z += beta * old.z;
            o.w += beta * old.w;
        }
        *reinterpret_cast<float4*>(xp) = o;
    }
    else
    {
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (iw0 + e < g.in[2])
                xp[e] = beta != 0.f ? alpha * acc[e] + beta * xp[e] : alpha * acc[e];
    }
}

// The same for windows of 3 with stride 2 and pad 1 along W (3 / stride 2 along H; WD = 3
// with stride 2 or 1 with stride 1 along D) and an even output row: cells 4t .. 4t+3 lie
// in the windows of outputs 2t, 2t+1 and 2t+2 only, so a thread loads two index bytes
// and two gradients in one access each and takes the third pair from its right-hand
// neighbour's registers; short rows share a block as in the forward kernel.  The sums
// run in the same order (D, H, then W ascending) as in the kernel above: same bits.
template <int WD>
__global__ void __launch_bounds__(POOL_THREADS)
    pool_bwd_index_w3s2_kernel(PoolGeom g, float alpha, float beta, const float* __restrict__ dy, float* dx,
                               const unsigned char* __restrict__ argmax, int tw_log2, long long rows)
{
    const int t = (blockIdx.y << tw_log2) + (threadIdx.x & ((1 << tw_log2) - 1));
    const long long row = (long long) blockIdx.x * (POOL_THREADS >> tw_log2) + (threadIdx.x >> tw_log2);
    if (row >= rows) // a warp never spans two rows: the whole warp leaves
        return;
    const int iw0 = 4 * t, ow0 = 2 * t;
    int ih, id;
    pool_split_row(row, rows, g.in[1], &id, &ih);
    const int c = blockIdx.z % g.c, n = blockIdx.z / g.c;
    const int sd = WD == 1 ? 1 : 2;
    int dlo, dhi, hlo, hhi;
    pool_cover(id, sd, g.pad[0], WD, g.out[0], &dlo, &dhi);
    pool_cover(ih, 2, g.pad[1], 3, g.out[1], &hlo, &hhi);
    if (id < g.lo[0] || id >= g.hi[0] || ih < g.lo[1] || ih >= g.hi[1])
        dhi = dlo - 1; // a row outside the global tensor is padding
    const int lane = threadIdx.x & 31;
    // offsets inside one (sample, channel) volume fit 32 bits (checked at the launch)
    const int ys0 = (int) g.ys[0], ys1 = (int) g.ys[1], astep = g.out[1] * g.out[2];
    const unsigned char* abase =
        argmax + ((size_t) n * g.c + c) * ((size_t) g.out[0] * astep) + ((dlo * g.out[1] + hlo) * g.out[2] + ow0);
    const float* dbase = dy + (size_t) n * g.ys_n + (size_t) c * g.ys_c + (dlo * ys0 + hlo * ys1 + ow0);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    const bool two = ow0 + 1 < g.out[2], third = ow0 + 2 < g.out[2];
    // at most two output planes and two output rows hold this input row: all their loads
    // are issued before the first is used (which of the four exist is the same for the
    // whole warp)
    constexpr int JD = WD == 1 ? 1 : 2;
    int a0[JD * 2], a1[JD * 2];
    float d0[JD * 2], d1[JD * 2];
#pragma unroll
    for (int jd = 0; jd < JD; ++jd)
#pragma unroll
        for (int jh = 0; jh < 2; ++jh)
        {
            const int k = jd * 2 + jh;
            // 255 is the index pass's "empty window" and never a tap
            a0[k] = a1[k] = 255;
            d0[k] = d1[k] = 0.f;
            if (dlo + jd <= dhi && hlo + jh <= hhi && two)
            {
                const uchar2 a = __ldg(reinterpret_cast<const uchar2*>(abase + (jd * astep + jh * g.out[2])));
                const float2 d = __ldg(reinterpret_cast<const float2*>(dbase + (jd * ys0 + jh * ys1)));
                a0[k] = a.x;
                a1[k] = a.y;
                d0[k] = d.x;
                d1[k] = d.y;
            }
        }
#pragma unroll
    for (int jd = 0; jd < JD; ++jd)
#pragma unroll
        for (int jh = 0; jh < 2; ++jh)
        {
            const int k = jd * 2 + jh;
            const int od = dlo + jd, oh = hlo + jh;
            if (od > dhi || oh > hhi)
                continue;
            int a2 = __shfl_down_sync(0xffffffffu, a0[k], 1);
            float d2 = __shfl_down_sync(0xffffffffu, d0[k], 1);
            if (lane == 31)
            {
                a2 = third ? (int) __ldg(abase + (jd * astep + jh * g.out[2] + 2)) : 255;
                d2 = third ? __ldg(dbase + (jd * ys0 + jh * ys1 + 2)) : 0.f;
            }
            // tap of window (od, oh, ow) at cell i: tb + i - (2 ow - 1)
            const int tb = ((id - (od * sd - g.pad[0])) * 3 + (ih - (oh * 2 - g.pad[1]))) * 3;
            if (a0[k] == tb + 1)
                acc[0] += d0[k];
            if (a0[k] == tb + 2)
                acc[1] += d0[k];
            if (a1[k] == tb)
                acc[1] += d1[k];
            if (a1[k] == tb + 1)
                acc[2] += d1[k];
            if (a1[k] == tb + 2)
                acc[3] += d1[k];
            if (a2 == tb)
                acc[3] += d2;
        }
    if (iw0 >= g.in[2])
        return;
    float* xp = dx + (size_t) n * g.xs_n + (size_t) c * g.xs_c + (id * (int) g.xs[0] + ih * (int) g.xs[1] + iw0);
    if (iw0 + 4 <= g.in[2] && (reinterpret_cast<uintptr_t>(xp) & 15) == 0)
    {
        float4 o = make_float4(alpha * acc[0], alpha * acc[1], alpha * acc[2], alpha * acc[3]);
        if (beta != 0.f)
        {
            const float4 old = *reinterpret_cast<const float4*>(xp);
            o.x += beta * old.x;
            o.y += beta * old.y;
            o.z += beta * old.z;
            o.w += beta * old.w;
        }
        *reinterpret_cast<float4*>(xp) = o;
    }
    else
    {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (iw0 + e < g.in[2])
                xp[e] = beta != 0.f ? alpha * acc[e] + beta * xp[e] : alpha * acc[e];
    }
}

// The same gather with pad 1 along H (and D, for WD = 3) as well: a thread owns the four
// cells in each row of a 2 x 2 block of input rows (planes 2p, 2p+1 x rows 2q, 2q+1; one
// plane for WD = 1).  Those rows lie in the windows of output planes p, p+1 and output
// rows q, q+1 only, at fixed taps (row 2q is tap 1 of window q; row 2q+1 tap 2 of
// window q and tap 0 of window q+1), so the index bytes and gradients of the 2 x 2
// window rows are loaded once for sixteen cells and every comparison is against a
// constant.  For WD = 3 the thread walks along D: window plane p+1 is kept for the next
// block, and the plane behind it is on its way while this one is compared (269 -> 258 us
// for 16 x 256^3; 190 us at the rate of a copy).  Cells outside the global tensor never
// were a window's maximum, so they need no mask.  Per cell the sums run in the same order
// (D, H, then W ascending).
struct PoolWindows
{
    int a[3];   // index byte of windows 2t, 2t+1, 2t+2 (255: no window)
    float d[3]; // their gradients
};

template <int WD>
__global__ void __launch_bounds__(POOL_THREADS)
    pool_bwd_index_block_kernel(PoolGeom g, float alpha, float beta, const float* __restrict__ dy, float* dx,
                                const unsigned char* __restrict__ argmax, int tw_log2, int blocks_h, long long rows,
                                int seg, int blocks_d)
{
    constexpr int JD = WD == 1 ? 1 : 2;
    const int t = (blockIdx.y << tw_log2) + (threadIdx.x & ((1 << tw_log2) - 1));
    const long long row = (long long) blockIdx.x * (POOL_THREADS >> tw_log2) + (threadIdx.x >> tw_log2);
    if (row >= rows) // a warp never spans two row blocks: the whole warp leaves
        return;
    const int iw0 = 4 * t, ow0 = 2 * t;
    int s, q;
    pool_split_row(row, rows, blocks_h, &s, &q);
    const int c = blockIdx.z % g.c, n = blockIdx.z / g.c;
    const int lane = threadIdx.x & 31;
    // offsets inside one (sample, channel) volume fit 32 bits (checked at the launch)
    const int ys0 = (int) g.ys[0], ys1 = (int) g.ys[1], astep = g.out[1] * g.out[2];
    const unsigned char* abase =
        argmax + ((size_t) n * g.c + c) * ((size_t) g.out[0] * astep) + (q * g.out[2] + ow0);
    const float* dbase = dy + (size_t) n * g.ys_n + (size_t) c * g.ys_c + (q * ys1 + ow0);
    const bool two = ow0 + 1 < g.out[2], third = ow0 + 2 < g.out[2];
    // rows q, q + 1 of window plane od: which exist is the same for the whole warp
    auto fetch = [&](int od, PoolWindows (&w)[2]) {
#pragma unroll
        for (int jh = 0; jh < 2; ++jh)
        {
            w[jh] = {{255, 255, 255}, {0.f, 0.f, 0.f}};
            if (od < g.out[0] && q + jh < g.out[1] && two)
            {
                const unsigned char* ap = abase + (od * astep + jh * g.out[2]);
                const float* dp = dbase + (od * ys0 + jh * ys1);
                const uchar2 a = __ldg(reinterpret_cast<const uchar2*>(ap));
                const float2 d = __ldg(reinterpret_cast<const float2*>(dp));
                w[jh].a[0] = a.x, w[jh].a[1] = a.y;
                w[jh].d[0] = d.x, w[jh].d[1] = d.y;
                if (lane == 31 && third)
                    w[jh].a[2] = __ldg(ap + 2), w[jh].d[2] = __ldg(dp + 2);
            }
        }
    };
    // window 2t+2 is the right-hand neighbour's first
    auto share = [&](PoolWindows (&w)[2]) {
#pragma unroll
        for (int jh = 0; jh < 2; ++jh)
        {
            const int a = __shfl_down_sync(0xffffffffu, w[jh].a[0], 1);
            const float d = __shfl_down_sync(0xffffffffu, w[jh].d[0], 1);
            if (lane != 31)
                w[jh].a[2] = a, w[jh].d[2] = d;
        }
    };
    float* xbase = dx + (size_t) n * g.xs_n + (size_t) c * g.xs_c;
    const int xs0 = (int) g.xs[0], xs1 = (int) g.xs[1];
    const int p0 = s * seg, p1 = min(p0 + seg, blocks_d);
    PoolWindows w[JD][2], ahead[2];
    fetch(p0, w[0]);
    if (JD == 2)
        fetch(p0 + 1, ahead);
    share(w[0]);
#pragma unroll 1
    for (int p = p0; p < p1; ++p)
    {
        if (JD == 2)
        {
            w[JD - 1][0] = ahead[0], w[JD - 1][1] = ahead[1];
            if (p + 1 < p1)
                fetch(p + 2, ahead);
            share(w[JD - 1]);
        }
#pragma unroll
        for (int pa = 0; pa < JD; ++pa)
#pragma unroll
            for (int rb = 0; rb < 2; ++rb)
            {
                const int id = JD == 2 ? 2 * p + pa : p, ih = 2 * q + rb;
                if (id >= g.in[0] || ih >= g.in[1] || iw0 >= g.in[2])
                    continue;
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int jd = 0; jd < JD; ++jd)
#pragma unroll
                    for (int jh = 0; jh < 2; ++jh)
                    {
                        // tap of input (plane pa, row rb) in window (jd, jh): coordinate - (2 * window - 1)
                        const int kd = JD == 2 ? pa - 2 * jd + 1 : 0, kh = rb - 2 * jh + 1;
                        if (kd < 0 || kd > 2 || kh < 0 || kh > 2)
                            continue;
                        const PoolWindows& v = w[jd][jh];
                        const int tb = (kd * 3 + kh) * 3; // tap at cell i of window ow: tb + i - (2 ow - 1)
                        if (v.a[0] == tb + 1)
                            acc[0] += v.d[0];
                        if (v.a[0] == tb + 2)
                            acc[1] += v.d[0];
                        if (v.a[1] == tb)
                            acc[1] += v.d[1];
                        if (v.a[1] == tb + 1)
                            acc[2] += v.d[1];
                        if (v.a[1] == tb + 2)
                            acc[3] += v.d[1];
                        if (v.a[2] == tb)
                            acc[3] += v.d[2];
                    }
                float* xp = xbase + (id * xs0 + ih * xs1 + iw0);
                if (iw0 + 4 <= g.in[2] && (reinterpret_cast<uintptr_t>(xp) & 15) == 0)
                {
                    float4 o = make_float4(alpha * acc[0], alpha * acc[1], alpha * acc[2], alpha * acc[3]);
                    if (beta != 0.f)
                    {
                        const float4 old = *reinterpret_cast<const float4*>(xp);
                        o.x += beta * old.x;
                        o.y += beta * old.y;
                        o.z += beta * old.z;
                        o.w += beta * old.w;
                    }
                    *reinterpret_cast<float4*>(xp) = o;
                }
                else
                {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (iw0 + e < g.in[2])
                            xp[e] = beta != 0.f ? alpha * acc[e] + beta * xp[e] : alpha * acc[e];
                }
            }
        if (JD == 2)
            w[0][0] = w[JD - 1][0], w[0][1] = w[JD - 1][1];
    }
}

// Outputs (or blocks) along D that one thread walks over: as many as leave the chip four
// times the blocks it holds, 16 at most (a walk re-reads one plane of its 2 * seg + 1).
int pool_walk(long long blocks_per_step, int steps)
{
    const long long seg = blocks_per_step * steps / ((long long) num_sms() * 8 * 4);
    return seg < 1 ? 1 : seg > 16 ? 16 : (int) seg;
}

int32_t pool_geom(const dcb_pool_desc* pd, const dcb_nd_desc* xd, const dcb_nd_desc* yd, PoolGeom* g)
{
    DCB_REQUIRE(pd && xd && yd, "null descriptor");
    DCB_REQUIRE(pd->nsd == 2 || pd->nsd == 3, "nsd must be 2 or 3");
    DCB_REQUIRE(xd->nsd == pd->nsd && yd->nsd == pd->nsd, "descriptor ranks do not match");
    DCB_REQUIRE(pd->mode == DCB_POOL_MAX || pd->mode == DCB_POOL_AVERAGE || pd->mode == DCB_POOL_AVERAGE_NO_PAD,
                "unknown pooling mode");
    DCB_REQUIRE(xd->n == yd->n && xd->c == yd->c, "sample / channel counts do not match");
    DCB_REQUIRE(xd->n >= 0 && xd->c >= 0 && xd->n * xd->c < (1ll << 31), "too many (n, c) planes");
    g->n = (int) xd->n;
    g->c = (int) xd->c;
    g->mode = pd->mode;
    for (int i = 0; i < 3; ++i)
    {
        DCB_REQUIRE(pd->window[i] >= 1 && pd->strides[i] >= 1 && pd->pads[i] >= 0, "bad window / stride / pad");
        DCB_REQUIRE(pd->pads[i] < pd->window[i], "a window entirely inside the padding");
        DCB_REQUIRE(xd->dims[i] < (1ll << 30) && yd->dims[i] < (1ll << 30), "extent too large");
        const long long span = xd->dims[i] + 2ll * pd->pads[i] - pd->window[i];
        DCB_REQUIRE(yd->dims[i] == (span < 0 ? 0 : span / pd->strides[i] + 1),
                    "output extent does not match input, pad, stride, window");
        g->in[i] = (int) xd->dims[i];
        g->out[i] = (int) yd->dims[i];
        g->win[i] = pd->window[i];
        g->pad[i] = pd->pads[i];
        g->stride[i] = pd->strides[i];
        g->xs[i] = xd->strides[i];
        g->ys[i] = yd->strides[i];
        DCB_REQUIRE(pd->outside_lo[i] >= 0 && pd->outside_hi[i] >= 0
                        && pd->outside_lo[i] + pd->outside_hi[i] <= xd->dims[i],
                    "outside_lo / outside_hi exceed the window");
        DCB_REQUIRE(pd->outside_lo[i] < pd->window[i] && pd->outside_hi[i] < pd->window[i],
                    "a window entirely inside the padding");
        g->lo[i] = pd->outside_lo[i];
        g->hi[i] = (int) xd->dims[i] - pd->outside_hi[i];
    }
    if (pd->nsd == 2)
        DCB_REQUIRE(pd->window[0] == 1 && pd->pads[0] == 0 && pd->strides[0] == 1, "slot 0 must be trivial for 2-D");
    DCB_REQUIRE(xd->strides[2] == 1 || xd->dims[2] <= 1, "W must be unit-stride");
    DCB_REQUIRE(yd->strides[2] == 1 || yd->dims[2] <= 1, "W must be unit-stride");
    g->xs_n = xd->sn;
    g->xs_c = xd->sc;
    g->ys_n = yd->sn;
    g->ys_c = yd->sc;
    return DCB_OK;
}

// grid.x carries (plane, row), the large product; grid.z (sample, channel)
bool pool_grid(int w, long long rows, long long planes, dim3* grid)
{
    const long long wt = (w + POOL_THREADS - 1) / POOL_THREADS;
    if (rows > 0x7fffffffll || wt > 65535 || planes > 65535)
        return false;
    *grid = dim3((unsigned) rows, (unsigned) wt, (unsigned) planes);
    return true;
}

// Picks the kernel instance whose compile-time window and stride match: cubic
// (or, for 2-D, square with a unit D slot) windows of 3 with stride 1 or 2 and of 2
// with stride 2; anything else runs the generic instance.
#define DCB_POOL_DISPATCH(g)                                                                                          \
    do                                                                                                                \
    {                                                                                                                 \
        const int w_ = (g).win[2], s_ = (g).stride[2];                                                               \
        const bool sq_ = (g).win[1] == w_ && (g).stride[1] == s_;                                                    \
        const bool flat_ = (g).win[0] == 1 && (g).stride[0] == 1;                                                    \
        const bool cube_ = (g).win[0] == w_ && (g).stride[0] == s_;                                                  \
        if (sq_ && cube_ && w_ == 3 && s_ == 2)                                                                       \
            DCB_POOL_CALL(3, 3, 2);                                                                                   \
        else if (sq_ && cube_ && w_ == 3 && s_ == 1)                                                                  \
            DCB_POOL_CALL(3, 3, 1);                                                                                   \
        else if (sq_ && cube_ && w_ == 2 && s_ == 2)                                                                  \
            DCB_POOL_CALL(2, 2, 2);                                                                                   \
        else if (sq_ && flat_ && w_ == 3 && s_ == 2)                                                                  \
            DCB_POOL_CALL(1, 3, 2);                                                                                   \
        else if (sq_ && flat_ && w_ == 3 && s_ == 1)                                                                  \
            DCB_POOL_CALL(1, 3, 1);                                                                                   \
        else if (sq_ && flat_ && w_ == 2 && s_ == 2)                                                                  \
            DCB_POOL_CALL(1, 2, 2);                                                                                   \
        else                                                                                                          \
            DCB_POOL_CALL(0, 0, 0);                                                                                   \
    } while (0)

template <int WD, int W, int S, int O>
void launch_pool_cells(const PoolGeom& g, float alpha, float beta, const float* x, float* y, unsigned char* argmax, long long rows,
                       unsigned planes, cudaStream_t stream)
{
    const int threads = (g.out[2] + O - 1) / O; // a row needs
    int tw_log2 = 8;
    while (tw_log2 > 2 && (1 << (tw_log2 - 1)) >= threads)
        --tw_log2;
    const long long rpb = POOL_THREADS >> tw_log2;
    // (as many blocks in x and y as the caller's grid has, or fewer)
    const dim3 grid((unsigned) ((rows + rpb - 1) / rpb), (unsigned) ((threads + (1 << tw_log2) - 1) >> tw_log2), planes);
    (g.mode == DCB_POOL_MAX ? pool_fwd_cells_kernel<WD, W, S, true, O> : pool_fwd_cells_kernel<WD, W, S, false, O>)
        <<<grid, POOL_THREADS, 0, stream>>>(g, alpha, beta, x, y, argmax, tw_log2, rows);
}

template <int WD, int W, int S>
void launch_pool_general(const PoolGeom& g, float alpha, float beta, const float* x, float* y, unsigned char* argmax, dim3 grid,
                         int tw_log2, long long rows, cudaStream_t stream)
{
    if constexpr (WD == 0)
        pool_fwd_kernel<<<grid, POOL_THREADS, 0, stream>>>(g, alpha, beta, x, y, argmax, tw_log2, rows);
    else
    {
        // Outputs a thread, us with 1 / 2 / 4 (maxima).  Few outputs: latency, 4 x 16^3, 3 / 1 3.9 / 4.3 /
        // 4.9, 4 x 93 x 19 x 57, 2 / 2 2.9 / 3.1 / 3.5.  Stride 1: what neighbours share, 16 x 64 x 100 x
        // 90, 3 / 1 199 / 173 / 133.  Stride 2: they share a cell or none, and two keep twice the threads
        // in flight, 4 x 58 x 108 x 238, 2 / 2 10.4 / 7.8 / 9.6, 3 / 2 17.6 / 13.3 / 19.9; but large tensors
        // of rows that do not fill a warp like that, 64 x 78 x 62 x 47, 2 / 2 26.7 / 19.5 / 16.4, 3 / 2, pad 1
        // 55.0 / 38.9 / 33.1.
        const long long outs = rows * g.out[2] * grid.z;
        if (outs <= 65536)
            launch_pool_cells<WD, W, S, 1>(g, alpha, beta, x, y, argmax, rows, grid.z, stream);
        else if (S > 1 && (outs < 300000 || g.out[2] >= 63))
            launch_pool_cells<WD, W, S, 2>(g, alpha, beta, x, y, argmax, rows, grid.z, stream);
        else
            launch_pool_cells<WD, W, S, 4>(g, alpha, beta, x, y, argmax, rows, grid.z, stream);
    }
}

template <int WD, int W, int S, int E, bool UNIFORM>
void launch_pool_bwd_cells(const PoolGeom& g, float alpha, float beta, const float* dy, float* dx, const unsigned char* idx, int tw_log2,
                           unsigned planes, cudaStream_t stream)
{
    const long long rows = (long long) g.in[0] * g.in[1], rpb = UNIFORM ? 1 : POOL_THREADS >> tw_log2;
    const int threads = (g.in[2] + E - 1) / E; // a row needs
    // (as many blocks in x and y as pool_grid has allowed, or fewer)
    const dim3 grid((unsigned) ((rows + rpb - 1) / rpb), (unsigned) ((threads + (1 << tw_log2) - 1) >> tw_log2), planes);
    (idx ? pool_bwd_cells_kernel<WD, W, S, true, E, UNIFORM> : pool_bwd_cells_kernel<WD, W, S, false, E, UNIFORM>)
        <<<grid, UNIFORM ? 1 << tw_log2 : POOL_THREADS, 0, stream>>>(g, alpha, beta, dy, dx, idx, tw_log2, rows);
}

template <int WD, int W, int S>
void launch_pool_bwd(const PoolGeom& g, float alpha, float beta, const float* dy, float* dx, const unsigned char* idx, unsigned planes,
                     cudaStream_t stream)
{
    // Few cells: one a thread, latency counts (us, one / four: averages of 4 x 32 x 32, 5 / 1 6.3 / 7.9;
    // 4 x 16^3, 3 / 1 6.3 / 8.3, maxima 8.1 / 10.4; but 4 x 32^3 10.3 / 8.7 and 13.1 / 11.5).
    const bool few = (long long) g.in[0] * g.in[1] * g.in[2] * planes <= 32768;
    const int threads = few ? g.in[2] : (g.in[2] + 3) / 4; // a row needs
    int tw_log2 = 8;
    while (tw_log2 > 2 && (1 << (tw_log2 - 1)) >= threads)
        --tw_log2;
    if (few)
        launch_pool_bwd_cells<WD, W, S, 1, false>(g, alpha, beta, dy, dx, idx, tw_log2, planes, stream);
    else if (W != 0 && tw_log2 >= 6)
        launch_pool_bwd_cells<WD, W, S, 4, W != 0>(g, alpha, beta, dy, dx, idx, tw_log2, planes, stream);
    else
        launch_pool_bwd_cells<WD, W, S, 4, false>(g, alpha, beta, dy, dx, idx, tw_log2, planes, stream);
}

int32_t launch_pool_fwd(const PoolGeom& g, float alpha, float beta, const float* x, float* y, unsigned char* argmax,
                        cudaStream_t stream)
{
    // the two-outputs-per-thread kernel: window 3, stride 2, pad 1 along W and H, the same or
    // a unit slot along D, input rows on 16-byte boundaries
    const bool flat = g.win[0] == 1 && g.stride[0] == 1;
    const bool cube = g.win[0] == 3 && g.stride[0] == 2;
    const bool pair = g.win[2] == 3 && g.stride[2] == 2 && g.pad[2] == 1 && g.win[1] == 3 && g.stride[1] == 2
                      && (flat || cube) && (reinterpret_cast<uintptr_t>(x) & 15) == 0 && g.xs[0] % 4 == 0
                      && g.xs[1] % 4 == 0 && g.xs_c % 4 == 0 && g.xs_n % 4 == 0 && g.out[2] >= 2
                      && (long long) g.out[0] * g.out[1] * g.out[2] < (1ll << 31)
                      && (g.out[0] - 1) * g.ys[0] + (g.out[1] - 1) * g.ys[1] + g.out[2] < (1ll << 31)
                      && (g.in[0] - 1) * g.xs[0] + (g.in[1] - 1) * g.xs[1] + g.in[2] < (1ll << 31);
    const int wcells = pair ? (g.out[2] + 1) / 2 : g.out[2]; // threads a row needs
    int tw_log2 = 8; // threads of a row per block: 32, 64, 128 or 256
    while (tw_log2 > 5 && (1 << (tw_log2 - 1)) >= wcells)
        --tw_log2;
    const long long tiles = (wcells + (1 << tw_log2) - 1) >> tw_log2;
    const long long rows = (long long) g.out[0] * g.out[1], planes = (long long) g.n * g.c;
    const long long rpb = POOL_THREADS >> tw_log2;
    const long long gx = (rows + rpb - 1) / rpb;
    if (gx > 0x7fffffffll || tiles > 65535 || planes > 65535)
    {
        set_last_error("tensor too large for the pooling grid");
        return DCB_UNSUPPORTED;
    }
    const dim3 grid((unsigned) gx, (unsigned) tiles, (unsigned) planes);
    if (pair && cube && g.lo[2] == 0 && g.hi[2] == g.in[2])
    {
        const int seg = pool_walk((g.out[1] + rpb - 1) / rpb * tiles * planes, g.out[0]);
        const long long mrows = (long long) ((g.out[0] + seg - 1) / seg) * g.out[1];
        const dim3 mgrid((unsigned) ((mrows + rpb - 1) / rpb), (unsigned) tiles, (unsigned) planes);
        auto kernel = g.mode != DCB_POOL_MAX ? pool_fwd_march_kernel<false, false>
                      : argmax               ? pool_fwd_march_kernel<true, true>
                                             : pool_fwd_march_kernel<true, false>;
        kernel<<<mgrid, POOL_THREADS, 0, stream>>>(g, alpha, beta, x, y, argmax, tw_log2, mrows, seg);
        DCB_LAUNCH_CHECK();
        return DCB_OK;
    }
    if (pair)
    {
        if (cube)
            pool_fwd_w3s2_kernel<3><<<grid, POOL_THREADS, 0, stream>>>(g, alpha, beta, x, y, argmax, tw_log2, rows);
        else
            pool_fwd_w3s2_kernel<1><<<grid, POOL_THREADS, 0, stream>>>(g, alpha, beta, x, y, argmax, tw_log2, rows);
        DCB_LAUNCH_CHECK();
        return DCB_OK;
    }
#define DCB_POOL_CALL(WD, W, S) launch_pool_general<WD, W, S>(g, alpha, beta, x, y, argmax, grid, tw_log2, rows, stream)
    DCB_POOL_DISPATCH(g);
#undef DCB_POOL_CALL
    DCB_LAUNCH_CHECK();
    return DCB_OK;
}

} // namespace
} // namespace dcb

using namespace dcb;

extern "C" int32_t dcb_pool_fwd(const dcb_pool_desc* pd, const dcb_nd_desc* xd, const dcb_nd_desc* yd, double alpha,
                                const void* x, double beta, void* y, void* stream)
{
    PoolGeom g;
    const int32_t st = pool_geom(pd, xd, yd, &g);
    if (st != DCB_OK)
        return st;
    if ((long long) g.n * g.c * g.out[0] * g.out[1] * g.out[2] == 0)
        return DCB_OK;
    DCB_REQUIRE(x && y, "null argument");
    return launch_pool_fwd(g, (float) alpha, (float) beta, static_cast<const float*>(x), static_cast<float*>(y),
                           nullptr, as_stream(stream));
}

extern "C" int64_t dcb_pool_bwd_workspace_bytes(const dcb_pool_desc* pd, const dcb_nd_desc* xd, const dcb_nd_desc* yd)
{
    PoolGeom g;
    if (pool_geom(pd, xd, yd, &g) != DCB_OK)
        return -1;
    if (g.mode != DCB_POOL_MAX || g.win[0] * g.win[1] * g.win[2] > 255)
        return 0;
    return (int64_t) g.n * g.c * g.out[0] * g.out[1] * g.out[2];
}

extern "C" int32_t dcb_pool_bwd(const dcb_pool_desc* pd, const dcb_nd_desc* xd, const dcb_nd_desc* yd, double alpha,
                                const void* y, const void* dy, const void* x, double beta, void* dx, void* workspace,
                                int64_t workspace_bytes, void* stream)
{
    PoolGeom g;
    const int32_t st = pool_geom(pd, xd, yd, &g);
    if (st != DCB_OK)
        return st;
    if ((long long) g.n * g.c * g.in[0] * g.in[1] * g.in[2] == 0)
        return DCB_OK;
    DCB_REQUIRE(dy && dx && (pd->mode != DCB_POOL_MAX || (x && y)), "null argument");
    dim3 grid;
    if (!pool_grid(g.in[2], (long long) g.in[0] * g.in[1], (long long) g.n * g.c, &grid))
    {
        set_last_error("tensor too large for the pooling grid");
        return DCB_UNSUPPORTED;
    }
    // With a workspace the position of every window's first maximum is worked out
    // first, by the forward kernel's separable pass (from x alone: nothing is kept
    // between calls), and the gather compares one byte per window instead of
    // scanning the window's earlier cells.
    const unsigned char* idx = nullptr;
    const int64_t need = dcb_pool_bwd_workspace_bytes(pd, xd, yd);
    if (g.mode == DCB_POOL_MAX && workspace && need > 0 && workspace_bytes >= need
        && (long long) g.n * g.c * g.out[0] * g.out[1] * g.out[2] > 0)
    {
        const int32_t st2 =
            launch_pool_fwd(g, 1.f, 0.f, static_cast<const float*>(x), nullptr, static_cast<unsigned char*>(workspace),
                            as_stream(stream));
        if (st2 != DCB_OK)
            return st2;
        idx = static_cast<const unsigned char*>(workspace);
    }
    const bool flat = g.win[0] == 1 && g.stride[0] == 1;
    const bool cube = g.win[0] == 3 && g.stride[0] == 2;
    const bool even = g.ys[0] % 2 == 0 && g.ys[1] % 2 == 0 && g.ys_c % 2 == 0 && g.ys_n % 2 == 0 && g.out[2] % 2 == 0
                      && (reinterpret_cast<uintptr_t>(dy) & 7) == 0 && (reinterpret_cast<uintptr_t>(idx) & 1) == 0;
    // offsets inside one (sample, channel) volume as 32-bit integers
    const bool small = (long long) g.out[0] * g.out[1] * g.out[2] < (1ll << 31)
                       && (g.out[0] - 1) * g.ys[0] + (g.out[1] - 1) * g.ys[1] + g.out[2] < (1ll << 31)
                       && (g.in[0] - 1) * g.xs[0] + (g.in[1] - 1) * g.xs[1] + g.in[2] < (1ll << 31);
    if (idx && g.win[2] == 3 && g.stride[2] == 2 && g.pad[2] == 1 && g.win[1] == 3 && g.stride[1] == 2
        && (flat || cube) && even && small)
    {
        const int wcells = (g.in[2] + 3) / 4; // threads a row needs
        int tw_log2 = 8;
        while (tw_log2 > 5 && (1 << (tw_log2 - 1)) >= wcells)
            --tw_log2;
        const long long tiles = (wcells + (1 << tw_log2) - 1) >> tw_log2;
        const long long rpb = POOL_THREADS >> tw_log2;
        // pad 1 along H (and D): a thread takes a 2 x 2 block of rows
        const bool block = g.pad[1] == 1 && (cube ? g.pad[0] == 1 : g.pad[0] == 0);
        if (block && tiles <= 65535)
        {
            const int blocks_h = (g.in[1] + 1) / 2;
            const int blocks_d = cube ? (g.in[0] + 1) / 2 : g.in[0];
            const int seg = cube ? pool_walk((blocks_h + rpb - 1) / rpb * tiles * grid.z, blocks_d) : 1;
            const long long brows = (long long) ((blocks_d + seg - 1) / seg) * blocks_h;
            const long long bgx = (brows + rpb - 1) / rpb;
            const dim3 gridb((unsigned) bgx, (unsigned) tiles, grid.z);
            if (cube)
                pool_bwd_index_block_kernel<3><<<gridb, POOL_THREADS, 0, as_stream(stream)>>>(
                    g, (float) alpha, (float) beta, static_cast<const float*>(dy), static_cast<float*>(dx), idx,
                    tw_log2, blocks_h, brows, seg, blocks_d);
            else
                pool_bwd_index_block_kernel<1><<<gridb, POOL_THREADS, 0, as_stream(stream)>>>(
                    g, (float) alpha, (float) beta, static_cast<const float*>(dy), static_cast<float*>(dx), idx,
                    tw_log2, blocks_h, brows, seg, blocks_d);
            DCB_LAUNCH_CHECK();
            return DCB_OK;
        }
        const long long rows = (long long) g.in[0] * g.in[1];
        const long long gx = (rows + rpb - 1) / rpb;
        if (gx <= 0x7fffffffll && tiles <= 65535)
        {
            const dim3 gridp((unsigned) gx, (unsigned) tiles, grid.z);
            if (cube)
                pool_bwd_index_w3s2_kernel<3><<<gridp, POOL_THREADS, 0, as_stream(stream)>>>(
                    g, (float) alpha, (float) beta, static_cast<const float*>(dy), static_cast<float*>(dx), idx,
                    tw_log2, rows);
            else
                pool_bwd_index_w3s2_kernel<1><<<gridp, POOL_THREADS, 0, as_stream(stream)>>>(
                    g, (float) alpha, (float) beta, static_cast<const float*>(dy), static_cast<float*>(dx), idx,
                    tw_log2, rows);
            DCB_LAUNCH_CHECK();
            return DCB_OK;
        }
    }
    if (idx || g.mode != DCB_POOL_MAX)
    {
#define DCB_POOL_CALL(WD, W, S)                                                                                       \
    launch_pool_bwd<WD, W, S>(g, (float) alpha, (float) beta, static_cast<const float*>(dy), static_cast<float*>(dx), idx, \
                              grid.z, as_stream(stream))
        DCB_POOL_DISPATCH(g);
#undef DCB_POOL_CALL
        DCB_LAUNCH_CHECK();
        return DCB_OK;
    }
#define DCB_POOL_CALL(WD, W, S)                                                                                       \
    pool_bwd_kernel<WD, W, S><<<grid, POOL_THREADS, 0, as_stream(stream)>>>(                                         \
        g, (float) alpha, (float) beta, static_cast<const float*>(y), static_cast<const float*>(dy),                  \
        static_cast<const float*>(x), static_cast<float*>(dx))
    DCB_POOL_DISPATCH(g);
#undef DCB_POOL_CALL
    DCB_LAUNCH_CHECK();
    return DCB_OK;
}
