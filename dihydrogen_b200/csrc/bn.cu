// Batch-normalisation kernels (and LeakyReLU): HBM-bound streaming kernels.
//
// Every (n, c) plane of an NC[D]HW window is a set of contiguous runs (see
// RunGeom).  A "unit" is up to 256 x (8 or 16) vector elements of one run, or,
// where runs are short (the rows of a shard with halo cells along W, whose
// pitch keeps them apart), several consecutive runs; blocks of channel c
// (blockIdx.y) stride over that channel's units with 16-byte vector accesses
// where the strides allow.
//
// Reductions are two-stage and fixed-order: each block writes its fp64 partial
// to scratch, the last block of a channel (ticket) folds the partials in index
// order, so results are reproducible run to run.  fp32 atomics, as the
// reference uses (batchnorm.cu:39-132), are not.
#include <atomic>

#include "common.cuh"

namespace dcb
{

constexpr int BN_THREADS = 256;
// Vector elements a thread has in flight per unit.  The streaming kernels (apply,
// backward apply, LeakyReLU) want many: 16 x 16 bytes per thread measured 0.341 ms
// for the 2 GiB of the bench layer's apply against 0.367 ms with 4; the reductions
// hold accumulators beside the data and are fastest with 8 (0.155 / 0.304 ms against
// 0.168 / 0.328 ms with 16).
constexpr int BN_UNROLL_MAP = 16;
constexpr int BN_UNROLL_RED = 8;
// ... and 16 where a vector element is one float, as in rows of odd length (2 x 24 x
// 67 x 83 x 101: statistics 34.9 -> 30.7 us, backward sums 57.8 -> 54.2 us).
template <int V>
constexpr int bn_unroll_red = V == 1 ? 2 * BN_UNROLL_RED : BN_UNROLL_RED;
// ... and 4 where vectors are pieces of unaligned runs (see Piece), or 8 (make_multi).
constexpr int BN_UNROLL_PIECES = 4;

struct UnitGeom
{
    RunGeom g;
    long long upr;   // units per run (1 when runs are packed)
    long long upc;   // units per channel
    int unit;        // scalars per unit = 256 * unroll * vector width
    // Packed short runs: a unit is up to rpu consecutive runs of one outer step,
    // vpr vector elements each.  Unpacked: rpu = 1, vpr = 0, magic = 0.
    int rpu, vpr;
    unsigned magic;  // ceil(2^32 / vpr): e / vpr = umulhi(e, magic) for the e < 4096 used here
    long long gpo;   // units per outer step
};

static UnitGeom make_units(const RunGeom& g, int vec, int unroll)
{
    const int BN_UNIT_VECS = BN_THREADS * unroll; // vector elements per unit
    UnitGeom u;
    u.g = g;
    u.unit = BN_UNIT_VECS * vec;
    u.upr = (g.len + u.unit - 1) / u.unit;
    u.upc = g.n * g.rows * u.upr;
    u.rpu = 1;
    u.vpr = 0;
    u.magic = 0;
    u.gpo = 0;
    const long long vpr = g.len / vec;
    if (g.rows_inner > 1 && vpr >= 2 && vpr * 2 <= BN_UNIT_VECS)
    {
        u.vpr = (int) vpr;
        u.rpu = (int) (BN_UNIT_VECS / vpr < g.rows_inner ? BN_UNIT_VECS / vpr : g.rows_inner);
        u.magic = (unsigned) ((0x100000000ull + (unsigned long long) vpr - 1) / (unsigned long long) vpr);
        u.gpo = (g.rows_inner + u.rpu - 1) / u.rpu;
        u.upr = 1;
        u.upc = g.n * (g.rows / g.rows_inner) * u.gpo;
    }
    return u;
}

struct UnitPos
{
    long long nn, row, e0;
    int count; // scalars in this unit (packed: in each of its runs)
    int nsub;  // runs in this unit
};

__device__ __forceinline__ UnitPos decode_unit(const UnitGeom& ug, long long u)
{
    UnitPos p;
    if (ug.vpr)
    {
        const long long grp = u % ug.gpo;
        const long long t = u / ug.gpo;
        const long long outers = ug.g.rows / ug.g.rows_inner;
        const long long first = grp * ug.rpu;
        p.row = (t % outers) * ug.g.rows_inner + first;
        p.nn = t / outers;
        p.e0 = 0;
        p.count = (int) ug.g.len;
        const long long left = ug.g.rows_inner - first;
        p.nsub = left < ug.rpu ? (int) left : ug.rpu;
        return p;
    }
    const long long chunk = u % ug.upr;
    const long long t = u / ug.upr;
    p.row = t % ug.g.rows;
    p.nn = t / ug.g.rows;
    p.e0 = chunk * ug.unit;
    const long long rem = ug.g.len - p.e0;
    p.count = rem < ug.unit ? (int) rem : ug.unit;
    p.nsub = 1;
    return p;
}

// Vector element e of a unit: which of the unit's runs it falls into and where.
struct ElemPos
{
    int sub, col;
    bool on;
    template <int V>
    __device__ __forceinline__ long long off(const RunStrides& s) const
    {
        return (long long) sub * s.s_inner + (long long) col * V;
    }
};

template <bool PACKED>
__device__ __forceinline__ ElemPos elem_pos(const UnitGeom& ug, const UnitPos& p, int e, int nv)
{
    ElemPos q;
    if (PACKED)
    {
        q.sub = (int) __umulhi((unsigned) e, ug.magic);
        q.col = e - q.sub * ug.vpr;
        q.on = q.sub < p.nsub;
    }
    else
    {
        q.sub = 0;
        q.col = e;
        q.on = e < nv;
    }
    return q;
}

__device__ __forceinline__ long long unit_offset(const RunStrides& s,
                                                 const RunGeom& g,
                                                 const UnitPos& p, int c)
{
    return p.nn * s.sn + (long long) c * s.sc
           + (p.row / g.rows_inner) * s.s_outer
           + (p.row % g.rows_inner) * s.s_inner + p.e0;
}

template <int V>
struct Vec;
template <>
struct Vec<1>
{
    float v[1];
    __device__ __forceinline__ void load(const float* p) { v[0] = *p; }
    __device__ __forceinline__ void store(float* p) const { *p = v[0]; }
};
template <>
struct Vec<2>
{
    float v[2];
    __device__ __forceinline__ void load(const float* p)
    {
        float2 t = *reinterpret_cast<const float2*>(p);
        v[0] = t.x;
        v[1] = t.y;
    }
    __device__ __forceinline__ void store(float* p) const
    {
        *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
    }
};
template <>
struct Vec<4>
{
    float v[4];
    __device__ __forceinline__ void load(const float* p)
    {
        float4 t = *reinterpret_cast<const float4*>(p);
        v[0] = t.x;
        v[1] = t.y;
        v[2] = t.z;
        v[3] = t.w;
    }
    __device__ __forceinline__ void store(float* p) const
    {
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
};

// Long runs whose starts are not 16-byte aligned (planes of odd size): the reductions read them
// in the aligned pieces of four that they lie in, all tensors of a call alike (pieces_fit).  Piece
// q of a run that starts `head` floats above a boundary is its elements 4 q - head onwards; those
// at the run's ends have fewer than four.
struct Piece
{
    long long e;
    int lo, hi; // of the piece's elements, those of the run
    __device__ __forceinline__ Piece(long long q, int head, long long len)
    {
        e = 4 * q - head;
        lo = e < 0 ? head : 0;
        hi = len - e < 4 ? (int) (len - e > 0 ? len - e : 0) : 4;
    }
    __device__ __forceinline__ bool any() const { return lo < hi; }
    // Element i of the four is the run's.
    __device__ __forceinline__ bool has(int i) const { return i >= lo && i < hi; }
    // Zeros stand for the others.  (Nothing is added up here: the loads of all of a thread's
    // pieces are in flight together.)
    __device__ __forceinline__ void load(const float* run, Vec<4>* v) const
    {
        if (lo == 0 && hi == 4)
            v->load(run + e);
        else
#pragma unroll
            for (int i = 0; i < 4; ++i)
                v->v[i] = has(i) ? run[e + i] : 0.f;
    }
};

// Sum NV doubles across the block; result valid in thread 0.
template <int NV>
__device__ __forceinline__ void block_reduce(double (&val)[NV])
{
    __shared__ double sm[NV][BN_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; ++i)
    {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            val[i] += __shfl_down_sync(0xffffffffu, val[i], o);
        if (lane == 0)
            sm[i][warp] = val[i];
    }
    __syncthreads();
    if (warp == 0)
    {
#pragma unroll
        for (int i = 0; i < NV; ++i)
        {
            double v = lane < BN_THREADS / 32 ? sm[i][lane] : 0.0;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1)
                v += __shfl_down_sync(0xffffffffu, v, o);
            val[i] = v;
        }
    }
    __syncthreads();
}

// Second stage: the last block of channel c folds NV x nblocks partials in
// index order and hands the totals to `emit` (thread 0).
template <int NV, typename Emit>
__device__ __forceinline__ void finish_channel(double (&val)[NV],
                                               double* partial,
                                               unsigned* tickets, Emit emit)
{
    const int c = blockIdx.y;
    const int nb = gridDim.x;
    __shared__ int last;
    if (threadIdx.x == 0)
    {
#pragma unroll
        for (int i = 0; i < NV; ++i)
            partial[((size_t) c * nb + blockIdx.x) * NV + i] = val[i];
        __threadfence();
        const unsigned prev = atomicAdd(&tickets[c], 1u);
        last = (prev == (unsigned) nb - 1);
    }
    __syncthreads();
    if (!last)
        return;
    __threadfence();
    if (threadIdx.x < 32)
    {
        double acc[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i)
            acc[i] = 0.0;
        // Lane l takes partials l, l+32, ... in order; lanes are then folded
        // by a fixed shuffle tree.
        for (int b = threadIdx.x; b < nb; b += 32)
#pragma unroll
            for (int i = 0; i < NV; ++i)
                acc[i] += partial[((size_t) c * nb + b) * NV + i];
#pragma unroll
        for (int i = 0; i < NV; ++i)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                acc[i] += __shfl_down_sync(0xffffffffu, acc[i], o);
        if (threadIdx.x == 0)
        {
            emit(acc);
            tickets[c] = 0;
        }
    }
}

// PIECES: the pieces of four that a thread has in flight, 0: aligned vectors
template <int V, bool PACKED, int PIECES = 0>
__global__ void __launch_bounds__(BN_THREADS)
    bn_stats_kernel(const float* __restrict__ x, RunStrides xs, UnitGeom ug,
                    double* partial, unsigned* tickets,
                    float* __restrict__ sums, float* __restrict__ sqsums)
{
    constexpr int U = PIECES ? PIECES : bn_unroll_red<V>;
    wait_for_previous_kernel(x);
    const int c = blockIdx.y;
    double acc[2] = {0.0, 0.0};
    for (long long u = blockIdx.x; u < ug.upc; u += gridDim.x)
    {
        const UnitPos p = decode_unit(ug, u);
        const float* xp = x + unit_offset(xs, ug.g, p, c);
        const int nv = p.count / V;
        Vec<V> v[U];
        bool on[U];
        float s = 0.f, q = 0.f;
        const float* run = xp - p.e0;
        const int head = (int) (reinterpret_cast<uintptr_t>(run) >> 2 & 3);
#pragma unroll
        for (int k = 0; k < U; ++k)
        {
            if (PIECES)
            {
                const Piece pc(p.e0 / 4 + threadIdx.x + k * BN_THREADS, head, ug.g.len);
                on[k] = pc.any();
                if constexpr (PIECES)
                    pc.load(run, &v[k]);
                continue;
            }
            const ElemPos ep = elem_pos<PACKED>(ug, p, threadIdx.x + k * BN_THREADS, nv);
            on[k] = ep.on;
            if (on[k])
                v[k].load(xp + ep.template off<V>(xs));
        }
#pragma unroll
        for (int k = 0; k < U; ++k)
        {
            if (on[k])
#pragma unroll
                for (int i = 0; i < V; ++i)
                {
                    s += v[k].v[i];
                    q = fmaf(v[k].v[i], v[k].v[i], q);
                }
            // (pieces: sums of sixteen in fp32, as element by element)
            if (k == U - 1 || (PIECES && k % BN_UNROLL_PIECES == BN_UNROLL_PIECES - 1))
            {
                acc[0] += (double) s;
                acc[1] += (double) q;
                s = q = 0.f;
            }
        }
    }
    block_reduce<2>(acc);
    finish_channel<2>(acc, partial, tickets, [&](const double(&t)[2]) {
        sums[c] = (float) t[0];
        sqsums[c] = (float) t[1];
    });
}

// Operation order of sums_to_statistics_functor (batchnorm.cu:297-312).
__device__ __forceinline__ void sums_to_statistics(long long num_per_sum, float& sum, float& sqsum)
{
    const float nps = (float) num_per_sum;
    const float m = sum / nps;
    const float sq = sqsum / nps;
    float v = sq - m * m;
    v = v > 0.f ? v : 0.f;
    v *= nps / (nps - 1.f);
    sum = m;
    sqsum = v;
}

// (one rounding fewer than written, wherever it is inlined)
__device__ __forceinline__ float running_update(float decay, float running, float value)
{
    return __fmaf_rn(decay, running, __fmul_rn(1.f - decay, value));
}

__global__ void bn_finalize_kernel(int channels, long long num_per_sum,
                                   float decay, float* mean, float* var,
                                   float* running_mean, float* running_var)
{
    wait_for_previous_kernel(mean, var, running_mean, running_var);
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= channels)
        return;
    if (num_per_sum > 0)
    {
        float m = mean[c], v = var[c];
        sums_to_statistics(num_per_sum, m, v);
        mean[c] = m;
        var[c] = v;
        running_mean[c] = running_update(decay, running_mean[c], m);
        running_var[c] = running_update(decay, running_var[c], v);
    }
    else
    {
        var[c] = 1.f;
    }
}

// What bn_finalize_kernel does, by the apply kernel itself: every block turns its
// channel's sums into statistics, and when all blocks of the channel, a cluster, have read
// the sums, the first one writes them back.  One launch less between a small layer's
// statistics and its output, and nothing kept between calls.
struct FinalizeArgs
{
    long long num_per_sum;
    float decay;
    float *mean, *var, *running_mean, *running_var; // sums in, statistics out
};
constexpr unsigned BN_CLUSTER_MAX = 8; // blocks of a cluster that every device grants

// LEAKY: the leaky ReLU that follows the batch-norm in the same pass
// (y > 0 ? y : slope * y), one trip through HBM instead of two.
template <int V, bool LEAKY, bool PACKED, bool FINALIZE>
__global__ void __launch_bounds__(BN_THREADS)
    bn_apply_kernel(const float* __restrict__ x, RunStrides xs,
                    float* __restrict__ y, RunStrides ys, UnitGeom ug,
                    const float* mean, const float* var,
                    const float* __restrict__ scale,
                    const float* __restrict__ bias, float eps, float slope,
                    FinalizeArgs fin)
{
    wait_for_previous_kernel(x, mean, var, scale, bias);
    const int c = blockIdx.y;
    float m, v0;
    if (FINALIZE)
    {
        // one thread reads the sums, so that it knows when the block has them
        __shared__ float stat[2];
        if (threadIdx.x == 0)
        {
            float a = fin.mean[c], b = fin.var[c];
            sums_to_statistics(fin.num_per_sum, a, b);
            stat[0] = a;
            stat[1] = b;
        }
        __syncthreads();
        m = stat[0];
        v0 = stat[1];
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    }
    else
    {
        m = mean[c];
        v0 = var[c];
    }
    const float inv_stdev = rsqrtf(v0 + eps);
    const float sc = scale[c], bi = bias[c];
    for (long long u = blockIdx.x; u < ug.upc; u += gridDim.x)
    {
        const UnitPos p = decode_unit(ug, u);
        const float* xp = x + unit_offset(xs, ug.g, p, c);
        float* yp = y + unit_offset(ys, ug.g, p, c);
        const int nv = p.count / V;
        Vec<V> v[BN_UNROLL_MAP];
        ElemPos ep[BN_UNROLL_MAP];
#pragma unroll
        for (int k = 0; k < BN_UNROLL_MAP; ++k)
        {
            ep[k] = elem_pos<PACKED>(ug, p, threadIdx.x + k * BN_THREADS, nv);
            if (ep[k].on)
                v[k].load(xp + ep[k].template off<V>(xs));
        }
#pragma unroll
        for (int k = 0; k < BN_UNROLL_MAP; ++k)
            if (ep[k].on)
            {
#pragma unroll
                for (int i = 0; i < V; ++i)
                {
                    const float xhat = (v[k].v[i] - m) * inv_stdev;
                    const float o = sc * xhat + bi;
                    v[k].v[i] = LEAKY ? (o > 0.f ? o : o * slope) : o;
                }
                v[k].store(yp + ep[k].template off<V>(ys));
            }
    }
    if (FINALIZE)
    {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (threadIdx.x == 0 && blockIdx.x == 0)
        {
            fin.mean[c] = m;
            fin.var[c] = v0;
            fin.running_mean[c] = running_update(fin.decay, fin.running_mean[c], m);
            fin.running_var[c] = running_update(fin.decay, fin.running_var[c], v0);
        }
    }
}

template <int V, bool PACKED, int PIECES = 0>
__global__ void __launch_bounds__(BN_THREADS)
    bn_bwd_reduce_kernel(const float* __restrict__ x, RunStrides xs,
                         const float* __restrict__ dy, RunStrides ds,
                         UnitGeom ug, const float* __restrict__ mean,
                         const float* __restrict__ var,
                         const float* __restrict__ scale, float eps,
                         double* partial, unsigned* tickets,
                         float* __restrict__ dscale, float* __restrict__ dbias,
                         float* __restrict__ dmean, float* __restrict__ dvar)
{
    constexpr int U = PIECES ? PIECES : bn_unroll_red<V>;
    wait_for_previous_kernel(x, dy, mean, var, scale);
    const int c = blockIdx.y;
    const float m = mean[c];
    const float sc = scale[c];
    const float inv_stdev = rsqrtf(var[c] + eps);
    const float dvar_factor = inv_stdev * inv_stdev * inv_stdev / 2;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (long long u = blockIdx.x; u < ug.upc; u += gridDim.x)
    {
        const UnitPos p = decode_unit(ug, u);
        const float* xp = x + unit_offset(xs, ug.g, p, c);
        const float* dp = dy + unit_offset(ds, ug.g, p, c);
        const int nv = p.count / V;
        Vec<V> vx[U], vd[U];
        bool on[U];
        float a[4] = {};
        auto add = [&](float xv, float g) {
            // backprop1 (batchnorm.cu:940-952)
            const float xhat = (xv - m) * inv_stdev;
            a[0] += g * xhat;
            a[1] += g;
            const float dxhat = g * sc;
            a[2] += -dxhat * inv_stdev;
            a[3] += -dxhat * (xv - m) * dvar_factor;
        };
        const float *xrun = xp - p.e0, *drun = dp - p.e0;
        const int head = (int) (reinterpret_cast<uintptr_t>(xrun) >> 2 & 3);
#pragma unroll
        for (int k = 0; k < U; ++k)
        {
            if (PIECES)
            {
                const Piece pc(p.e0 / 4 + threadIdx.x + k * BN_THREADS, head, ug.g.len);
                on[k] = pc.any();
                if constexpr (PIECES)
                {
                    pc.load(xrun, &vx[k]);
                    pc.load(drun, &vd[k]);
                }
                continue;
            }
            const ElemPos ep = elem_pos<PACKED>(ug, p, threadIdx.x + k * BN_THREADS, nv);
            on[k] = ep.on;
            if (on[k])
            {
                vx[k].load(xp + ep.template off<V>(xs));
                vd[k].load(dp + ep.template off<V>(ds));
            }
        }
#pragma unroll
        for (int k = 0; k < U; ++k)
            if (on[k])
            {
                const Piece pc(p.e0 / 4 + threadIdx.x + k * BN_THREADS, head, ug.g.len);
#pragma unroll
                for (int i = 0; i < V; ++i)
                    if (!PIECES || pc.has(i)) // (an infinite mean times a zero that stands for no element is none)
                        add(vx[k].v[i], vd[k].v[i]);
            }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            acc[i] += (double) a[i];
    }
    block_reduce<4>(acc);
    finish_channel<4>(acc, partial, tickets, [&](const double(&t)[4]) {
        dscale[c] = (float) t[0];
        dbias[c] = (float) t[1];
        dmean[c] = (float) t[2];
        dvar[c] = (float) t[3];
    });
}

// Goes through the tensors from their end: the reduction went through them forwards, so
// what it read last is still in L2, and the backward filter finds the beginning there
// (backward pass of 256^3 x 16 channels: 3190 us forwards, 3153 us like this).
template <int V, bool PACKED>
__global__ void __launch_bounds__(BN_THREADS)
    bn_bwd_apply_kernel(const float* x, RunStrides xs,
                        const float* __restrict__ dy, RunStrides ds, float* dx,
                        RunStrides os, UnitGeom ug,
                        const float* __restrict__ mean,
                        const float* __restrict__ var,
                        const float* __restrict__ scale,
                        const float* __restrict__ dmean,
                        const float* __restrict__ dvar, float eps,
                        long long num_per_sum)
{
    wait_for_previous_kernel(x, dy, mean, var, scale, dmean, dvar);
    const int c = gridDim.y - 1 - blockIdx.y; // the last one first, as the units below
    const float m = mean[c];
    const float sc = scale[c];
    const float inv_stdev = rsqrtf(var[c] + eps);
    // backprop2 (batchnorm.cu:1333-1335)
    const float dmean_term = dmean[c] / (float) num_per_sum;
    const float dvar_term = dvar[c] * 2 / (float) (num_per_sum - 1);
    for (long long u = ug.upc - 1 - blockIdx.x; u >= 0; u -= gridDim.x)
    {
        const UnitPos p = decode_unit(ug, u);
        const float* xp = x + unit_offset(xs, ug.g, p, c);
        const float* dp = dy + unit_offset(ds, ug.g, p, c);
        float* op = dx + unit_offset(os, ug.g, p, c);
        const int nv = p.count / V;
        Vec<V> vx[BN_UNROLL_MAP], vd[BN_UNROLL_MAP];
        ElemPos ep[BN_UNROLL_MAP];
#pragma unroll
        for (int k = 0; k < BN_UNROLL_MAP; ++k)
        {
            ep[k] = elem_pos<PACKED>(ug, p, threadIdx.x + k * BN_THREADS, nv);
            if (ep[k].on)
            {
                vx[k].load(xp + ep[k].template off<V>(xs));
                vd[k].load(dp + ep[k].template off<V>(ds));
            }
        }
#pragma unroll
        for (int k = 0; k < BN_UNROLL_MAP; ++k)
            if (ep[k].on)
            {
#pragma unroll
                for (int i = 0; i < V; ++i)
                {
                    const float dxhat = vd[k].v[i] * sc;
                    float r = dxhat * inv_stdev;
                    r += dmean_term;
                    r += dvar_term * (vx[k].v[i] - m);
                    vd[k].v[i] = r;
                }
                vd[k].store(op + ep[k].template off<V>(os));
            }
    }
}

// mode 0: y = x>0 ? x : slope*x ;  mode 1: dx = x>0 ? dy : slope*dy
template <int V, int MODE, bool PACKED>
__global__ void __launch_bounds__(BN_THREADS)
    leaky_relu_kernel(const float* x, RunStrides xs,
                      const float* __restrict__ dy, RunStrides ds, float* out,
                      RunStrides os, UnitGeom ug, float slope)
{
    wait_for_previous_kernel(x, dy);
    const int c = blockIdx.y;
    for (long long u = blockIdx.x; u < ug.upc; u += gridDim.x)
    {
        const UnitPos p = decode_unit(ug, u);
        const float* xp = x + unit_offset(xs, ug.g, p, c);
        const float* dp = MODE ? dy + unit_offset(ds, ug.g, p, c) : nullptr;
        float* op = out + unit_offset(os, ug.g, p, c);
        const int nv = p.count / V;
#pragma unroll
        for (int k = 0; k < BN_UNROLL_MAP; ++k)
        {
            const ElemPos ep = elem_pos<PACKED>(ug, p, threadIdx.x + k * BN_THREADS, nv);
            if (ep.on)
            {
                Vec<V> vx, vd;
                vx.load(xp + ep.template off<V>(xs));
                if (MODE)
                    vd.load(dp + ep.template off<V>(ds));
#pragma unroll
                for (int i = 0; i < V; ++i)
                {
                    const float src = MODE ? vd.v[i] : vx.v[i];
                    vx.v[i] = vx.v[i] > 0.f ? src : slope * src;
                }
                vx.store(op + ep.template off<V>(os));
            }
        }
    }
}

static dim3 bn_grid(const UnitGeom& ug)
{
    long long per_c = (long long) num_sms() * 8 / (ug.g.c > 0 ? ug.g.c : 1);
    if (per_c < 1)
        per_c = 1;
    long long bx = ug.upc < per_c ? ug.upc : per_c;
    if (bx < 1)
        bx = 1;
    return dim3((unsigned) bx, (unsigned) ug.g.c);
}

// Common level / vector width for a set of same-shaped tensors.
struct MultiView
{
    UnitGeom ug;
    RunStrides s[3];
    int vec;
    int pieces; // reductions: aligned pieces of four (see Piece), so many a thread
};

// Whether all tensors' runs start equally far above a 16-byte boundary.
static bool pieces_fit(const MultiView& mv, const void* const* ptrs, int count)
{
    const RunStrides& a = mv.s[0];
    for (int i = 1; i < count; ++i)
    {
        const RunStrides& b = mv.s[i];
        const long long differ = (a.sn - b.sn) | (a.sc - b.sc) | (a.s_inner - b.s_inner) | (a.s_outer - b.s_outer);
        if ((differ & 3) != 0 || ((reinterpret_cast<uintptr_t>(ptrs[0]) ^ reinterpret_cast<uintptr_t>(ptrs[i])) & 15) != 0)
            return false;
    }
    return true;
}

static int32_t make_multi(const dcb_nd_desc* const* descs,
                          const void* const* ptrs, int count, MultiView* mv, int unroll, int unroll1,
                          bool reduction = false)
{
    int level = 2;
    for (int i = 0; i < count; ++i)
    {
        int32_t st = check_nd_desc(descs[i]);
        if (st != DCB_OK)
            return st;
        DCB_REQUIRE(same_extents(*descs[0], *descs[i]),
                    "tensor extents differ");
        const int l = run_level(*descs[i]);
        if (l < 0)
        {
            set_last_error("innermost dimension must have unit stride");
            return DCB_UNSUPPORTED;
        }
        level = l < level ? l : level;
    }
    RunGeom g;
    int vec = 4;
    for (int i = 0; i < count; ++i)
    {
        make_runs(*descs[i], level, &g, &mv->s[i]);
        const int v = run_vec(g, mv->s[i], ptrs[i]);
        vec = v < vec ? v : vec;
    }
    mv->ug = make_units(g, vec, vec == 1 ? unroll1 : unroll);
    mv->vec = vec;
    // Pieces, us element by element / with eight a thread / with four, with inputs that have left L2
    // (in brackets: with those that have not):
    //   statistics     2 x 24 x 67 x 83 x 101  38.9 / 30.7 / -    (28.0 / 19.1 / 22.8)
    //                  8 x 128 x 41 x 67       14.4 / 14.4 / 12.3 (8.4 / 8.5 / 6.5)
    //                  16 x 256 x 33 x 33      24.5 / 30.7 / 20.5 (14.7 / 20.2 / 15.1)
    //   backward sums  2 x 24 x 67 x 83 x 101  60.4 / 57.3 / 53.3 (44.2 / 43.6 / 38.1)
    //                  8 x 128 x 3 x 67 x 83   46.0 / 49.2 / 40.9 (33.1 / 39.0 / 29.1)
    //                  16 x 32 x 3 x 67 x 83   31.6 / 32.8 / 27.7 (16.2 / 21.5 / 17.0)
    //                  16 x 128 x 41 x 51      22.5 / 34.8 / 22.5 (13.0 / 23.8 / 13.7)
    //                  16 x 256 x 33 x 33      26.7 / 53.2 / 29.7 (19.1 / 38.5 / 20.8)
    // Shorter runs are mostly their ends.  The backward sums never take eight: 107 registers, two blocks
    // an SM (four: 60).  The statistics do where two thirds of such a unit's threads have work.
    mv->pieces = reduction && vec == 1 && mv->ug.vpr == 0 && g.len >= (count == 1 ? 1024 : 2048) && pieces_fit(*mv, ptrs, count)
                     ? BN_UNROLL_PIECES
                     : 0;
    if (mv->pieces)
    {
        const long long n = (g.len + 6) / 4, large = BN_THREADS * 2 * BN_UNROLL_PIECES;
        if (count == 1 && 3 * n >= 2 * large * ((n + large - 1) / large))
            mv->pieces = 2 * BN_UNROLL_PIECES;
        const long long unit = BN_THREADS * mv->pieces;
        mv->ug.unit = (int) unit * 4;
        mv->ug.upr = (n + unit - 1) / unit;
        mv->ug.upc = g.n * g.rows * mv->ug.upr;
    }
    DCB_REQUIRE(g.c <= 65535, "too many channels");
    return DCB_OK;
}

} // namespace dcb

using namespace dcb;

struct dcb_bn_plan
{
    dcb_nd_desc xd;
    double* partial = nullptr;
    unsigned* tickets = nullptr;
    int max_blocks = 0;
};

// PACKED (several short runs per unit) is a template parameter: the kernels that
// walk long runs keep their plain indexing.
#define DCB_VEC_DISPATCH(vec, packed, CALL)                                    \
    do                                                                         \
    {                                                                          \
        if (packed)                                                            \
        {                                                                      \
            if ((vec) == 4)                                                    \
            {                                                                  \
                CALL(4, true);                                                 \
            }                                                                  \
            else if ((vec) == 2)                                               \
            {                                                                  \
                CALL(2, true);                                                 \
            }                                                                  \
            else                                                               \
            {                                                                  \
                CALL(1, true);                                                 \
            }                                                                  \
        }                                                                      \
        else if ((vec) == 4)                                                   \
        {                                                                      \
            CALL(4, false);                                                    \
        }                                                                      \
        else if ((vec) == 2)                                                   \
        {                                                                      \
            CALL(2, false);                                                    \
        }                                                                      \
        else                                                                   \
        {                                                                      \
            CALL(1, false);                                                    \
        }                                                                      \
    } while (0)

extern "C" {

int32_t dcb_bn_plan_create(const dcb_nd_desc* xd, dcb_bn_plan** out)
{
    int32_t st = check_nd_desc(xd);
    if (st != DCB_OK)
        return st;
    DCB_REQUIRE(out != nullptr, "null argument");
    DCB_REQUIRE(xd->c > 0 && xd->c <= 65535, "channel count out of range");
    auto* p = new dcb_bn_plan();
    p->xd = *xd;
    p->max_blocks = num_sms() * 8;
    const size_t nb = (size_t) p->max_blocks + (size_t) xd->c;
    if (cudaMalloc(&p->partial, nb * 4 * sizeof(double)) != cudaSuccess
        || cudaMalloc(&p->tickets, (size_t) xd->c * sizeof(unsigned))
               != cudaSuccess
        || cudaMemset(p->tickets, 0, (size_t) xd->c * sizeof(unsigned))
               != cudaSuccess)
    {
        set_last_error("cudaMalloc of batch-norm scratch failed");
        (void) cudaGetLastError();
        cudaFree(p->partial);
        cudaFree(p->tickets);
        delete p;
        return DCB_CUDA_ERROR;
    }
    *out = p;
    return DCB_OK;
}

int32_t dcb_bn_plan_destroy(dcb_bn_plan* p)
{
    if (!p)
        return DCB_OK;
    cudaFree(p->partial);
    cudaFree(p->tickets);
    delete p;
    return DCB_OK;
}

int32_t dcb_bn_stats(dcb_bn_plan* plan, const void* x, void* sums,
                     void* sqsums, void* stream)
{
    DCB_REQUIRE(plan && x && sums && sqsums, "null argument");
    const dcb_nd_desc* descs[1] = {&plan->xd};
    const void* ptrs[1] = {x};
    MultiView mv;
    int32_t st = make_multi(descs, ptrs, 1, &mv, BN_UNROLL_RED, bn_unroll_red<1>, true);
    if (st != DCB_OK)
        return st;
    if (mv.ug.upc == 0)
    {
        DCB_CUDA_TRY(cudaMemsetAsync(sums, 0, plan->xd.c * sizeof(float),
                                     as_stream(stream)));
        DCB_CUDA_TRY(cudaMemsetAsync(sqsums, 0, plan->xd.c * sizeof(float),
                                     as_stream(stream)));
        return DCB_OK;
    }
    const dim3 grid = bn_grid(mv.ug);
#define CALL(VV, ...)                                                               \
    DCB_CUDA_TRY(launch_overlapped((bn_stats_kernel<VV, __VA_ARGS__>), grid, BN_THREADS, 0, as_stream(stream),           \
        static_cast<const float*>(x), mv.s[0], mv.ug, plan->partial,           \
        plan->tickets, static_cast<float*>(sums), static_cast<float*>(sqsums)))
    if (mv.pieces == BN_UNROLL_PIECES)
    {
        CALL(4, false, BN_UNROLL_PIECES);
    }
    else if (mv.pieces)
    {
        CALL(4, false, 2 * BN_UNROLL_PIECES);
    }
    else
        DCB_VEC_DISPATCH(mv.vec, mv.ug.vpr != 0, CALL);
#undef CALL
    DCB_LAUNCH_CHECK();
    return DCB_OK;
}

int32_t dcb_bn_finalize(int32_t channels, int64_t num_per_sum, float decay,
                        void* mean, void* var, void* running_mean,
                        void* running_var, void* stream)
{
    DCB_REQUIRE(channels > 0, "channels must be positive");
    DCB_REQUIRE(mean && var && running_mean && running_var, "null argument");
    DCB_CUDA_TRY(launch_overlapped(bn_finalize_kernel, dim3((unsigned) ((channels + 127) / 128)), 128, 0,
                                   as_stream(stream),
        channels, num_per_sum, decay, static_cast<float*>(mean),
        static_cast<float*>(var), static_cast<float*>(running_mean),
        static_cast<float*>(running_var)));
    DCB_LAUNCH_CHECK();
    return DCB_OK;
}

static int32_t bn_apply_impl(const dcb_nd_desc* xd, const void* x, const void* mean, const void* var,
                             const void* scale, const void* bias, float eps, bool leaky, float slope,
                             const dcb_nd_desc* yd, void* y, void* stream, const FinalizeArgs* fin = nullptr)
{
    DCB_REQUIRE(x && y && mean && var && scale && bias, "null argument");
    const dcb_nd_desc* descs[2] = {xd, yd};
    const void* ptrs[2] = {x, y};
    MultiView mv;
    int32_t st = make_multi(descs, ptrs, 2, &mv, BN_UNROLL_MAP, BN_UNROLL_MAP);
    if (st != DCB_OK)
        return st;
    if (mv.ug.upc == 0)
        return DCB_OK;
    const dim3 grid = bn_grid(mv.ug);
    if (fin && grid.x > BN_CLUSTER_MAX)
    {
        // too many blocks for a cluster, and enough work to hide a launch
        st = dcb_bn_finalize((int32_t) xd->c, fin->num_per_sum, fin->decay, fin->mean, fin->var, fin->running_mean,
                             fin->running_var, stream);
        if (st != DCB_OK)
            return st;
        fin = nullptr;
    }
    const FinalizeArgs f = fin ? *fin : FinalizeArgs();
#define CALL(VV, PP)                                                                                               \
    {                                                                                                              \
        auto kernel = leaky ? (fin ? bn_apply_kernel<VV, true, PP, true> : bn_apply_kernel<VV, true, PP, false>)   \
                            : (fin ? bn_apply_kernel<VV, false, PP, true> : bn_apply_kernel<VV, false, PP, false>); \
        DCB_CUDA_TRY(launch_overlapped_cluster(kernel, grid, fin ? grid.x : 1, BN_THREADS, 0, as_stream(stream),                               \
            static_cast<const float*>(x), mv.s[0], static_cast<float*>(y), mv.s[1], mv.ug,                         \
            static_cast<const float*>(mean), static_cast<const float*>(var), static_cast<const float*>(scale),     \
            static_cast<const float*>(bias), eps, slope, f));                                                       \
    }
    DCB_VEC_DISPATCH(mv.vec, mv.ug.vpr != 0, CALL);
#undef CALL
    DCB_LAUNCH_CHECK();
    return DCB_OK;
}

int32_t dcb_bn_finalize_apply(dcb_bn_plan* plan, int64_t num_per_sum, float decay, void* mean, void* var,
                              void* running_mean, void* running_var, const dcb_nd_desc* xd, const void* x,
                              const void* scale, const void* bias, float eps, float slope, const dcb_nd_desc* yd, void* y,
                              void* stream)
{
    DCB_REQUIRE(running_mean && running_var && num_per_sum > 0, "null argument");
    int32_t st = check_nd_desc(xd);
    if (st != DCB_OK)
        return st;
    DCB_REQUIRE((!plan || xd->c == plan->xd.c) && xd->n * xd->dims[0] * xd->dims[1] * xd->dims[2] > 0,
                "the plan is for another channel count, or the shard is empty");
    const FinalizeArgs f = {num_per_sum, decay, static_cast<float*>(mean), static_cast<float*>(var),
                            static_cast<float*>(running_mean), static_cast<float*>(running_var)};
    return bn_apply_impl(xd, x, mean, var, scale, bias, eps, slope != 1.f, slope, yd, y, stream, &f);
}

int32_t dcb_bn_apply(const dcb_nd_desc* xd, const void* x, const void* mean,
                     const void* var, const void* scale, const void* bias,
                     float eps, const dcb_nd_desc* yd, void* y, void* stream)
{
    return bn_apply_impl(xd, x, mean, var, scale, bias, eps, false, 1.f, yd, y, stream);
}

int32_t dcb_bn_apply_leaky_relu(const dcb_nd_desc* xd, const void* x,
                                const void* mean, const void* var,
                                const void* scale, const void* bias, float eps,
                                float slope, const dcb_nd_desc* yd, void* y,
                                void* stream)
{
    return bn_apply_impl(xd, x, mean, var, scale, bias, eps, true, slope, yd, y, stream);
}

int32_t dcb_bn_bwd_reduce(dcb_bn_plan* plan, const void* x,
                          const dcb_nd_desc* dyd, const void* dy,
                          const void* mean, const void* var, const void* scale,
                          float eps, void* dscale, void* dbias, void* dmean,
                          void* dvar, void* stream)
{
    DCB_REQUIRE(plan && x && dy && mean && var && scale && dscale && dbias
                    && dmean && dvar,
                "null argument");
    const dcb_nd_desc* descs[2] = {&plan->xd, dyd};
    const void* ptrs[2] = {x, dy};
    MultiView mv;
    int32_t st = make_multi(descs, ptrs, 2, &mv, BN_UNROLL_RED, bn_unroll_red<1>, true);
    if (st != DCB_OK)
        return st;
    if (mv.ug.upc == 0)
    {
        for (void* v : {dscale, dbias, dmean, dvar})
            DCB_CUDA_TRY(cudaMemsetAsync(v, 0, plan->xd.c * sizeof(float),
                                         as_stream(stream)));
        return DCB_OK;
    }
    const dim3 grid = bn_grid(mv.ug);
#define CALL(VV, ...)                                                               \
    DCB_CUDA_TRY(launch_overlapped((bn_bwd_reduce_kernel<VV, __VA_ARGS__>), grid, BN_THREADS, 0, as_stream(stream),      \
        static_cast<const float*>(x), mv.s[0], static_cast<const float*>(dy),  \
        mv.s[1], mv.ug, static_cast<const float*>(mean),                       \
        static_cast<const float*>(var), static_cast<const float*>(scale), eps, \
        plan->partial, plan->tickets, static_cast<float*>(dscale),             \
        static_cast<float*>(dbias), static_cast<float*>(dmean),                \
        static_cast<float*>(dvar)))
    if (mv.pieces)
    {
        CALL(4, false, BN_UNROLL_PIECES);
    }
    else
        DCB_VEC_DISPATCH(mv.vec, mv.ug.vpr != 0, CALL);
#undef CALL
    DCB_LAUNCH_CHECK();
    return DCB_OK;
}

int32_t dcb_bn_bwd_apply(const dcb_nd_desc* xd, const void* x,
                         const dcb_nd_desc* dyd, const void* dy,
                         const void* mean, const void* var, const void* scale,
                         const void* dmean, const void* dvar, float eps,
                         int64_t num_per_sum, const dcb_nd_desc* dxd, void* dx,
                         void* stream)
{
    DCB_REQUIRE(x && dy && dx && mean && var && scale && dmean && dvar,
                "null argument");
    const dcb_nd_desc* descs[3] = {xd, dyd, dxd};
    const void* ptrs[3] = {x, dy, dx};
    MultiView mv;
    int32_t st = make_multi(descs, ptrs, 3, &mv, BN_UNROLL_MAP, BN_UNROLL_MAP);
    if (st != DCB_OK)
        return st;
    if (mv.ug.upc == 0)
        return DCB_OK;
    const dim3 grid = bn_grid(mv.ug);
#define CALL(VV, PP)                                                               \
    DCB_CUDA_TRY(launch_overlapped((bn_bwd_apply_kernel<VV, PP>), grid, BN_THREADS, 0, as_stream(stream),       \
        static_cast<const float*>(x), mv.s[0], static_cast<const float*>(dy),  \
        mv.s[1], static_cast<float*>(dx), mv.s[2], mv.ug,                      \
        static_cast<const float*>(mean), static_cast<const float*>(var),       \
        static_cast<const float*>(scale), static_cast<const float*>(dmean),    \
        static_cast<const float*>(dvar), eps, (long long) num_per_sum))
    DCB_VEC_DISPATCH(mv.vec, mv.ug.vpr != 0, CALL);
#undef CALL
    DCB_LAUNCH_CHECK();
    return DCB_OK;
}

int32_t dcb_leaky_relu_fwd(const dcb_nd_desc* xd, const void* x, float slope,
                           const dcb_nd_desc* yd, void* y, void* stream)
{
    DCB_REQUIRE(x && y, "null argument");
    const dcb_nd_desc* descs[2] = {xd, yd};
    const void* ptrs[2] = {x, y};
    MultiView mv;
    int32_t st = make_multi(descs, ptrs, 2, &mv, BN_UNROLL_MAP, BN_UNROLL_MAP);
    if (st != DCB_OK)
        return st;
    if (mv.ug.upc == 0)
        return DCB_OK;
    const dim3 grid = bn_grid(mv.ug);
#define CALL(VV, PP)                                                               \
    DCB_CUDA_TRY(launch_overlapped((leaky_relu_kernel<VV, 0, PP>), grid, BN_THREADS, 0, as_stream(stream),      \
        static_cast<const float*>(x), mv.s[0], nullptr, mv.s[0],               \
        static_cast<float*>(y), mv.s[1], mv.ug, slope))
    DCB_VEC_DISPATCH(mv.vec, mv.ug.vpr != 0, CALL);
#undef CALL
    DCB_LAUNCH_CHECK();
    return DCB_OK;
}

int32_t dcb_leaky_relu_bwd(const dcb_nd_desc* xd, const void* x,
                           const dcb_nd_desc* dyd, const void* dy, float slope,
                           const dcb_nd_desc* dxd, void* dx, void* stream)
{
    DCB_REQUIRE(x && dy && dx, "null argument");
    const dcb_nd_desc* descs[3] = {xd, dyd, dxd};
    const void* ptrs[3] = {x, dy, dx};
    MultiView mv;
    int32_t st = make_multi(descs, ptrs, 3, &mv, BN_UNROLL_MAP, BN_UNROLL_MAP);
    if (st != DCB_OK)
        return st;
    if (mv.ug.upc == 0)
        return DCB_OK;
    const dim3 grid = bn_grid(mv.ug);
#define CALL(VV, PP)                                                               \
    DCB_CUDA_TRY(launch_overlapped((leaky_relu_kernel<VV, 1, PP>), grid, BN_THREADS, 0, as_stream(stream),      \
        static_cast<const float*>(x), mv.s[0], static_cast<const float*>(dy),  \
        mv.s[1], static_cast<float*>(dx), mv.s[2], mv.ug, slope))
    DCB_VEC_DISPATCH(mv.vec, mv.ug.vpr != 0, CALL);
#undef CALL
    DCB_LAUNCH_CHECK();
    return DCB_OK;
}

} // extern "C"

// ---------------------------------------------------------------------------
// Per-channel statistics without any device allocation.
//
// Some hosts cannot let a library call cudaMalloc: a training framework whose
// caching allocator already owns the whole device, code that runs between
// cudaStreamBeginCapture and EndCapture (allocation is illegal there), or a
// latency-critical loop where cudaMalloc's implicit device synchronisation is
// not acceptable.  For them this variant of dcb_bn_stats keeps its reduction
// scratch (per-block partial sums and the per-channel arrival tickets) in a
// fixed array that is part of the library image.  Every GPU that loads the
// library carries the array until the process exits.
// ---------------------------------------------------------------------------
namespace
{
constexpr int NOALLOC_MAX_CHANNELS = 1024;
constexpr int NOALLOC_MAX_BLOCKS = 4096; // blocks of one launch, all channels together
constexpr size_t NOALLOC_TICKET_BYTES = NOALLOC_MAX_CHANNELS * sizeof(unsigned);
constexpr size_t NOALLOC_PARTIAL_BYTES = (size_t) NOALLOC_MAX_BLOCKS * 2 * sizeof(double);
constexpr int NOALLOC_MAX_DEVICES = 64;

// Layout: [tickets: 1024 x u32][partials: 4096 x 2 x f64] = 68 KiB.
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_TICKET_BYTES + NOALLOC_PARTIAL_BYTES];

// Device address of the array on each device, resolved on first use.  In host
// code the symbol itself is only a handle, never a pointer a kernel may use.
// Host threads may race on an entry: they would all store the same address,
// so relaxed atomics are enough.
static std::atomic<void*> g_noalloc_addr[NOALLOC_MAX_DEVICES] = {};
} // namespace

extern "C" int32_t dcb_bn_stats_noalloc(const dcb_nd_desc* xd, const void* x, void* sums, void* sqsums,
                                        void* stream)
{
    DCB_REQUIRE(xd && x && sums && sqsums, "null argument");
    const dcb_nd_desc* descs[1] = {xd};
    const void* ptrs[1] = {x};
    MultiView mv;
    int32_t st = make_multi(descs, ptrs, 1, &mv, BN_UNROLL_RED, bn_unroll_red<1>, true);
    if (st != DCB_OK)
        return st;
    if (xd->c < 1 || xd->c > NOALLOC_MAX_CHANNELS)
    {
        set_last_error("dcb_bn_stats_noalloc handles 1..1024 channels; use dcb_bn_stats with a plan beyond that");
        return DCB_UNSUPPORTED;
    }
    int dev = 0;
    DCB_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES)
    {
        set_last_error("dcb_bn_stats_noalloc: device ordinal beyond 63");
        return DCB_UNSUPPORTED;
    }
    void* addr = g_noalloc_addr[dev].load(std::memory_order_relaxed);
    if (addr == nullptr)
    {
        // once per device, with that device current
        DCB_CUDA_TRY(cudaGetSymbolAddress(&addr, g_noalloc_scratch));
        g_noalloc_addr[dev].store(addr, std::memory_order_relaxed);
    }
    unsigned char* base = static_cast<unsigned char*>(addr);
    unsigned* tickets = reinterpret_cast<unsigned*>(base);
    double* partial = reinterpret_cast<double*>(base + NOALLOC_TICKET_BYTES);
    if (mv.ug.upc == 0)
    {
        DCB_CUDA_TRY(cudaMemsetAsync(sums, 0, xd->c * sizeof(float), as_stream(stream)));
        DCB_CUDA_TRY(cudaMemsetAsync(sqsums, 0, xd->c * sizeof(float), as_stream(stream)));
        return DCB_OK;
    }
    dim3 grid = bn_grid(mv.ug);
    // stay inside the fixed scratch: fewer blocks per channel if need be
    if ((long long) grid.x * grid.y > NOALLOC_MAX_BLOCKS)
        grid.x = (unsigned) (NOALLOC_MAX_BLOCKS / grid.y);
    if (grid.x < 1)
    {
        set_last_error("dcb_bn_stats_noalloc: launch does not fit the fixed scratch");
        return DCB_UNSUPPORTED;
    }
    // The array keeps whatever the previous call (or an interrupted one) left:
    // the arrival tickets must start at zero.  Partials are overwritten.
    DCB_CUDA_TRY(cudaMemsetAsync(tickets, 0, xd->c * sizeof(unsigned), as_stream(stream)));
#define CALL(VV, ...)                                                               \
    DCB_CUDA_TRY(launch_overlapped((bn_stats_kernel<VV, __VA_ARGS__>), grid, BN_THREADS, 0, as_stream(stream),           \
        static_cast<const float*>(x), mv.s[0], mv.ug, partial, tickets,        \
        static_cast<float*>(sums), static_cast<float*>(sqsums)))
    if (mv.pieces == BN_UNROLL_PIECES)
    {
        CALL(4, false, BN_UNROLL_PIECES);
    }
    else if (mv.pieces)
    {
        CALL(4, false, 2 * BN_UNROLL_PIECES);
    }
    else
        DCB_VEC_DISPATCH(mv.vec, mv.ug.vpr != 0, CALL);
#undef CALL
    DCB_LAUNCH_CHECK();
    return DCB_OK;
}
