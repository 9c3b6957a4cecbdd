// Re-distribution of a tensor between two block decompositions (sample-parallel
// <-> spatially partitioned, or any other pair): stands in for
// tensor::TensorMPICUDAShuffler
// (legacy/include/distconv/tensor/shuffle_mpi_cuda.hpp:14-512), which packs per
// destination rank, runs an MPI all-to-all-v through host-visible buffers and
// unpacks.
//
// Here every rank owns a receive window (IPC-mapped by its peers) shaped like
// its destination block, dense, W fastest, twice (consecutive shuffles
// alternate).  One kernel per rank, `put`, walks the intersections of the
// rank's source block with every destination block and stores the cells
// straight into the owners' windows (NVLink peer stores; the local part is an
// ordinary copy), then release-stores its epoch into a flag per destination.
// A second kernel, `wait_unpack`, waits (bounded) for the epochs of all ranks
// that hold a part of its block and copies the window into the destination
// tensor, skipping its halo.  No host staging, no collective call; ranks may
// run at most one shuffle apart, as with the halo exchange.
//
// HBM-bound: 8 B per cell at the sender (read + peer write), 8 B at the
// receiver (window read + tensor write).
#include "common.cuh"
#include "dcb.h"

#include <algorithm>
#include <cstring>
#include <vector>

#include <unistd.h>

namespace dcb
{
namespace
{

constexpr int SHF_THREADS = 256;
// Accesses of a thread in flight: 4, and 2 pieces, which are up to four loads each (us there and
// back, 2 ranks, with 4 and with 2: aligned rows 2 x 16 x 128^3 392 and 441, 2 x 16 x 206 x 32 x 120
// 175 and 204; in pieces 2 x 16 x 56 x 189 x 38 166 and 141, 2 x 16 x 77 x 91 x 45 203 and 153).
template <int WAY>
constexpr int shf_unroll = WAY == 2 ? 2 : 4;
constexpr long long SHF_MAX_CELLS = 2000000000ll;
constexpr int SHF_MAX_RANKS = 64;
constexpr size_t SHF_HEADER = 1024; // 64 flags, ticket, status

// How a job's cells are moved: one by one, by four where everything is a multiple of 16 bytes,
// or in the pieces that lie on 16-byte boundaries of the destination: loads as wide as
// the source allows, one 16-byte store, a place decoded once for four cells (two ranks, there and
// back, one by one / in pieces: 2 x 16 x 56 x 189 x 38 split along H 260 / 141 us, 2 x 4 x 232 x 69
// x 60 along W 189 / 128).
enum ShfAccess : int
{
    SHF_CELL = 0,
    SHF_VEC = 1,
    SHF_PIECE = 2
};
// Runs of fewer cells go one by one: a piece is a slot of a thread, and a run of L cells has
// up to (L + 6) / 4 of them.
constexpr long long SHF_PIECE_MIN = 6;

__host__ __device__ __forceinline__ int shf_way(int vec, long long len, int aligned)
{
    return vec && aligned ? SHF_VEC : (len >= SHF_PIECE_MIN ? SHF_PIECE : SHF_CELL);
}

// One box to move: `rows` runs of `len` contiguous cells.  Dimensions that are
// contiguous on both sides have been merged into the run.  Row r decodes into
// (i1, i2, i3, i4) over ext[1..4]; its first cell sits at
// a_off + sum i_k * a_stride[k] on the strided side and at
// b_off + sum i_k * b_stride[k] on the dense side.
struct ShfJob
{
    long long rows, len;
    long long ext[4];
    long long a_off, a_stride[4];
    long long b_off, b_stride[4];
    float* peer;            // put: the destination's window (parity 0)
    long long parity_pitch; // put: floats between the two halves of that window
    uint32_t* flag;         // put: flag to publish there; wait: own flag to wait on
    int vec;                // 16-byte accesses: offsets, strides and run allow them (if the bases do)
    // per way of access (ShfAccess)
    int split[3];           // long runs: a unit's accesses are of one run; else of the job
    long long units[3];
    long long per_run[3];   // accesses of a run
    FastDiv by_run[3], by_ext[4];
};

// Windows are unpacked from their end, where what was written last may still be in L2, by streaming
// stores, which leave it there, if the windows of this device's ranks together take three quarters of L2
// or more. Below, a window that is read from its start by plain stores leaves the tensor in L2 for its next
// reader. us, one way and a pass over the tensor behind it, rank's window from the start / from the end
// (B200, L2 of 126 MB; 2 x 16 x D x 128 x 128 split along D):
//   one rank on the device   34 MB 36.3 / 37.8, 67 MB 61.8 / 65.0, 84 MB 78.0 / 79.7, 101 MB 98.9 / 94.5, 134 MB 136.9 / 126.1
//   two ranks, of each       34 MB 85.8 / 91.9, 42 MB 101.2 / 108.2, 50 MB 121.7 / 121.6, 59 MB 142.9 / 138.0, 134 MB 281.6 / 276.8
// Either alone is 1 to 3 % slower than neither; pieces lose with both. (Not timed with a device per rank: one rank
// with a window of its own stands for it.)
inline bool shf_from_the_end(double window_bytes, double l2_bytes)
{
    return window_bytes >= 0.75 * l2_bytes;
}

struct ShfArgs
{
    const ShfJob* jobs;
    int njobs;
    float* tensor;
    float* window; // wait_unpack: own window of this parity
    int aligned;   // tensor starts on a 16-byte boundary (windows always do)
    int parity;    // put: which half of the destination windows
    uint32_t epoch;
    uint32_t* ticket;
    int* status;
    long long budget_ns;
};

// Where access n of a job is (or, split, access e0 of run r onwards): its run's first cells.
struct ShfRun
{
    const float* from;
    float* to;
};

__device__ __forceinline__ ShfRun shf_run(const ShfJob& j, uint32_t r, const float* from, float* to, const long long* fs,
                                          const long long* ts)
{
#pragma unroll
    for (int q = 0; q < 4; ++q)
    {
        const uint32_t d = j.by_ext[q].div(r), i = r - d * j.by_ext[q].d;
        r = d;
        from += (long long) i * fs[q];
        to += (long long) i * ts[q];
    }
    return {from, to};
}

// The cells e + lo .. e + hi - 1 of a run that are its piece q, where the run starts `head` cells
// above a boundary.
struct ShfRange
{
    long long e;
    int lo, hi;
};

__host__ __device__ __forceinline__ ShfRange shf_range(int head, long long q, long long len)
{
    const long long e = 4 * q - head;
    return {e, e < 0 ? head : 0, len - e < 4 ? (int) (len - e > 0 ? len - e : 0) : 4};
}

// Piece q of a run: up to four cells, from the 16-byte boundary of the destination that is q
// pieces above the one at or below the run's first cell.  Loads, then (put) the stores.
struct ShfPiece
{
    float v[4];
    float* to;
    int lo, hi; // cells lo .. hi - 1 of the piece exist

    __device__ __forceinline__ void get(const ShfRun& run, long long q, long long len)
    {
        const ShfRange r = shf_range((int) (reinterpret_cast<uintptr_t>(run.to) >> 2 & 3), q, len);
        const float* from = run.from + r.e;
        to = run.to + r.e;
        lo = r.lo;
        hi = r.hi;
        if (lo == 0 && hi == 4)
        {
            const int at = (int) (reinterpret_cast<uintptr_t>(from) >> 2 & 3);
            if (at == 0)
            {
                const float4 f = __ldcs(reinterpret_cast<const float4*>(from));
                v[0] = f.x, v[1] = f.y, v[2] = f.z, v[3] = f.w;
                return;
            }
            if (at == 2)
            {
                const float2 f = __ldcs(reinterpret_cast<const float2*>(from)), h = __ldcs(reinterpret_cast<const float2*>(from) + 1);
                v[0] = f.x, v[1] = f.y, v[2] = h.x, v[3] = h.y;
                return;
            }
        }
        // (cached: the lanes' cells of one load share sectors with those of the next)
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i >= lo && i < hi)
                v[i] = from[i];
    }
    __device__ __forceinline__ void none() { lo = hi = 0; }
    template <bool>
    __device__ __forceinline__ void put() const
    {
        if (lo == 0 && hi == 4)
        {
            *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]);
            return;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i >= lo && i < hi)
                to[i] = v[i];
    }
};

template <class T>
struct ShfCell
{
    T v;
    T* to;
    __device__ __forceinline__ void get(const ShfRun& run, long long e, long long)
    {
        to = reinterpret_cast<T*>(run.to) + e;
        v = __ldcs(reinterpret_cast<const T*>(run.from) + e);
    }
    __device__ __forceinline__ void none() { to = nullptr; }
    template <bool STREAM>
    __device__ __forceinline__ void put() const
    {
        if (to == nullptr)
            return;
        if (STREAM)
            __stcs(to, v);
        else
            *to = v;
    }
};

template <int WAY, bool STREAM, class T>
__device__ __forceinline__ void shf_unit(const ShfJob& j, long long u, const float* from, float* to, const long long* fs,
                                         const long long* ts)
{
    T a[shf_unroll<WAY>];
    constexpr int CHUNK = SHF_THREADS * shf_unroll<WAY>; // accesses of a unit
    if (j.split[WAY])
    {
        // CHUNK accesses of one long run
        const long long cpr = (j.per_run[WAY] + CHUNK - 1) / CHUNK;
        const long long r = u / cpr, e0 = (u - r * cpr) * CHUNK;
        const ShfRun run = shf_run(j, (uint32_t) r, from, to, fs, ts);
#pragma unroll
        for (int k = 0; k < shf_unroll<WAY>; ++k)
        {
            const long long e = e0 + threadIdx.x + k * SHF_THREADS;
            if (e < j.per_run[WAY])
                a[k].get(run, e, j.len);
            else
                a[k].none();
        }
    }
    else
    {
        const long long total = j.rows * j.per_run[WAY];
#pragma unroll
        for (int k = 0; k < shf_unroll<WAY>; ++k)
        {
            const long long n = u * CHUNK + threadIdx.x + k * SHF_THREADS;
            if (n < total)
            {
                const uint32_t r = j.by_run[WAY].div((uint32_t) n);
                a[k].get(shf_run(j, r, from, to, fs, ts), (uint32_t) n - r * j.by_run[WAY].d, j.len);
            }
            else
                a[k].none();
        }
    }
#pragma unroll
    for (int k = 0; k < shf_unroll<WAY>; ++k)
        a[k].template put<STREAM>();
}

// PUT: tensor (strided) -> peers' windows (dense).  !PUT: own window -> tensor.
// A unit is SHF_THREADS x shf_unroll accesses, all loads of a thread before its stores.  A warp per
// W run, decoded with eight run-time divisions and one access in flight per lane, took
// 100 us for 134 MB.
// PIECES: some job of the call takes them (a kernel of its own: with their registers the others took
// 5 us more of 50).
// BACK: see shf_from_the_end.
template <bool PUT, bool PIECES, bool BACK>
__global__ void __launch_bounds__(SHF_THREADS) shuffle_kernel(ShfArgs a)
{
    if (!PUT)
    {
        __shared__ int ok;
        if (threadIdx.x == 0)
        {
            ok = 1;
            for (int q = 0; q < a.njobs && ok; ++q)
                ok = bounded_wait_epoch(a.jobs[q].flag, a.epoch, a.budget_ns) ? 1 : 0;
        }
        __syncthreads();
        if (!ok)
        {
            if (threadIdx.x == 0)
                atomicExch(a.status, (int) DCB_PEER_TIMEOUT);
            return;
        }
    }
    __shared__ ShfJob j;
    long long u = blockIdx.x;
    for (int n = 0; n < a.njobs; ++n)
    {
        const int q = BACK ? a.njobs - 1 - n : n;
        __syncthreads();
        for (int i = threadIdx.x; i < (int) (sizeof(ShfJob) / 4); i += SHF_THREADS)
            reinterpret_cast<uint32_t*>(&j)[i] = reinterpret_cast<const uint32_t*>(&a.jobs[q])[i];
        __syncthreads();
        const int way = shf_way(j.vec, j.len, a.aligned);
        float* w = PUT ? j.peer + a.parity * j.parity_pitch : a.window;
        const long long* fs = PUT ? j.a_stride : j.b_stride;
        const long long* ts = PUT ? j.b_stride : j.a_stride;
        const float* from = (PUT ? a.tensor : w) + (PUT ? j.a_off : j.b_off);
        float* to = (PUT ? w : a.tensor) + (PUT ? j.b_off : j.a_off);
        for (; u < j.units[way]; u += gridDim.x)
        {
            const long long unit = BACK ? j.units[way] - 1 - u : u;
            if (way == SHF_VEC)
                shf_unit<SHF_VEC, BACK, ShfCell<float4>>(j, unit, from, to, fs, ts);
            else if (PIECES && way == SHF_PIECE)
                shf_unit<SHF_PIECE, BACK, ShfPiece>(j, unit, from, to, fs, ts);
            else
                shf_unit<SHF_CELL, BACK, ShfCell<float>>(j, unit, from, to, fs, ts);
        }
        u -= j.units[way];
    }
    if (PUT)
    {
        // the last block to arrive release-stores the epoch at every destination
        __syncthreads();
        if (threadIdx.x == 0 && last_block(a.ticket, gridDim.x))
            for (int q = 0; q < a.njobs; ++q)
                st_release_sys(a.jobs[q].flag, a.epoch);
    }
}

// Merges what is contiguous on both sides into the run and derives how the job is
// walked.
void finish_job(ShfJob* j)
{
    int n = 0;
    long long ext[4], as[4], bs[4];
    bool run = true;
    for (int k = 0; k < 4; ++k)
    {
        if (j->ext[k] == 1)
            continue;
        if (run && j->a_stride[k] == j->len && j->b_stride[k] == j->len)
        {
            j->len *= j->ext[k];
            continue;
        }
        run = false;
        if (n > 0 && j->a_stride[k] == as[n - 1] * ext[n - 1] && j->b_stride[k] == bs[n - 1] * ext[n - 1])
        {
            ext[n - 1] *= j->ext[k];
            continue;
        }
        ext[n] = j->ext[k], as[n] = j->a_stride[k], bs[n] = j->b_stride[k];
        ++n;
    }
    long long mix = j->len | j->a_off | j->b_off;
    j->rows = 1;
    for (int k = 0; k < 4; ++k)
    {
        j->ext[k] = k < n ? ext[k] : 1;
        j->a_stride[k] = k < n ? as[k] : 0;
        j->b_stride[k] = k < n ? bs[k] : 0;
        j->rows *= j->ext[k];
        mix |= j->a_stride[k] | j->b_stride[k];
        j->by_ext[k] = FastDiv::of((uint32_t) j->ext[k]);
    }
    j->vec = (mix & 3) == 0;
    for (int w = 0; w < 3; ++w)
    {
        j->per_run[w] = w == SHF_PIECE ? (j->len + 6) / 4 : j->len / (w == SHF_VEC ? 4 : 1);
        j->by_run[w] = FastDiv::of(j->per_run[w] > 0 && j->per_run[w] < (1 << 30) ? (uint32_t) j->per_run[w] : 1u);
        const long long chunk = SHF_THREADS * (w == SHF_PIECE ? shf_unroll<SHF_PIECE> : shf_unroll<SHF_VEC>);
        // Runs of at least two units, so that at most a third of a run's threads are idle in its last
        // one, or (one run) too many accesses for 31-bit indices.  By this way's own accesses: with
        // the cells of a run in pieces counted instead, 2 x 16 x 96 x 90 x 47 along H (runs of 2115)
        // took 204 us there and back, like this 160; runs of 3355 234 and 216, from 3969 on the same.
        j->split[w] = j->per_run[w] >= 2 * chunk || j->rows * j->len >= SHF_MAX_CELLS;
        j->units[w] = j->split[w] ? j->rows * ((j->per_run[w] + chunk - 1) / chunk) : (j->rows * j->per_run[w] + chunk - 1) / chunk;
    }
}

// Adds a job, in pieces of fewer than SHF_MAX_CELLS cells: inside one, indices and extents have
// 31 bits.  (A job of 2.9e9 cells in runs of 500 otherwise took a block per run.)
void add_jobs(ShfJob j, std::vector<ShfJob>* out, long long* units)
{
    long long cells = j.len;
    int outer = 0;
    for (int k = 0; k < 4; ++k)
    {
        cells *= j.ext[k];
        if (j.ext[k] > 1)
            outer = k;
    }
    if (cells >= SHF_MAX_CELLS && j.ext[outer] > 1)
    {
        ShfJob rest = j;
        j.ext[outer] /= 2;
        rest.ext[outer] -= j.ext[outer];
        j.rows = rest.rows = 0; // (finish_job counts them)
        rest.a_off += j.ext[outer] * j.a_stride[outer];
        rest.b_off += j.ext[outer] * j.b_stride[outer];
        add_jobs(j, out, units);
        add_jobs(rest, out, units);
        return;
    }
    finish_job(&j);
    out->push_back(j);
    *units += j.units[shf_way(j.vec, j.len, 1)];
}

struct ShfBlob
{
    WindowBlob win;
    uint32_t rank;
    uint32_t reserved;
    uint64_t parity_floats;
};
static_assert(sizeof(ShfBlob) <= DCB_SHUFFLE_BLOB_BYTES, "blob too large");

struct Box
{
    long long off[DCB_MAX_DIMS], ext[DCB_MAX_DIMS];
    long long volume() const
    {
        long long v = 1;
        for (int i = 0; i < DCB_MAX_DIMS; ++i)
            v *= ext[i];
        return v;
    }
};

Box to_box(const dcb_box& b, int nd)
{
    Box r;
    for (int i = 0; i < DCB_MAX_DIMS; ++i)
    {
        r.off[i] = i < nd ? b.off[i] : 0;
        r.ext[i] = i < nd ? b.ext[i] : 1;
    }
    return r;
}

bool intersect(const Box& a, const Box& b, Box* out)
{
    for (int i = 0; i < DCB_MAX_DIMS; ++i)
    {
        const long long lo = a.off[i] > b.off[i] ? a.off[i] : b.off[i];
        const long long ha = a.off[i] + a.ext[i], hb = b.off[i] + b.ext[i];
        const long long hi = ha < hb ? ha : hb;
        if (hi <= lo)
            return false;
        out->off[i] = lo;
        out->ext[i] = hi - lo;
    }
    return true;
}

} // namespace
} // namespace dcb

using namespace dcb;

struct dcb_shuffle_plan
{
    int nd, rank, nranks;
    dcb_tensor_desc src, dst;
    std::vector<Box> src_boxes, dst_boxes;
    Window win;
    long long parity_floats;
    std::vector<PeerMapping> peer_map; // by rank; only the destinations of my cells are opened
    ShfJob* d_put = nullptr;
    ShfJob* d_wait = nullptr;
    int n_put = 0, n_wait = 0;
    long long put_units = 0, wait_units = 0;
    bool put_pieces[2] = {}, wait_pieces[2] = {}; // whether a job takes pieces; by whether the tensor is 16-byte aligned
    bool from_the_end = false;
    uint32_t epoch = 0;
    bool connected = false;

    uint32_t* flags() { return reinterpret_cast<uint32_t*>(win.base); }
    uint32_t* ticket() { return flags() + SHF_MAX_RANKS; }
    int* status() { return reinterpret_cast<int*>(flags() + SHF_MAX_RANKS + 1); }
    float* window() { return reinterpret_cast<float*>(static_cast<char*>(win.base) + SHF_HEADER); }
};

namespace
{
int32_t check_shard(const dcb_tensor_desc* d, const Box& mine, int nd)
{
    DCB_REQUIRE(d->ndims == nd && d->dtype == DCB_F32, "descriptor rank / type");
    const long long vol = mine.volume();
    for (int i = 0; i < nd; ++i)
    {
        DCB_REQUIRE(d->real_shape[i] == d->local_shape[i] + 2ll * d->overlap[i], "real shape != local + 2 * overlap");
        // a rank that is not the root of a replicated dimension passes an empty box
        DCB_REQUIRE(vol == 0 || mine.ext[i] == d->local_shape[i], "this rank's box does not match its shard");
    }
    DCB_REQUIRE(d->pitch == 0 || d->pitch >= d->real_shape[0], "row pitch shorter than a row");
    return DCB_OK;
}

// element strides of the halo-extended shard, dimension 0 fastest
void real_strides(const dcb_tensor_desc& d, long long* s)
{
    long long acc = 1;
    for (int i = 0; i < DCB_MAX_DIMS; ++i)
    {
        s[i] = acc;
        acc *= i < d.ndims ? (i == 0 ? row_pitch(d) : d.real_shape[i]) : 1;
    }
}
} // namespace

extern "C" {

int32_t dcb_shuffle_plan_create(const dcb_tensor_desc* src, const dcb_tensor_desc* dst, const dcb_box* src_boxes,
                                const dcb_box* dst_boxes, int32_t rank, int32_t nranks, dcb_shuffle_plan** out)
{
    DCB_REQUIRE(src && dst && src_boxes && dst_boxes && out, "null argument");
    DCB_REQUIRE(nranks >= 1 && nranks <= SHF_MAX_RANKS && rank >= 0 && rank < nranks, "rank / nranks out of range");
    DCB_REQUIRE(src->ndims == dst->ndims && (src->ndims == 4 || src->ndims == 5), "ndims must be 4 or 5");
    const int nd = src->ndims;
    auto* p = new dcb_shuffle_plan();
    p->nd = nd;
    p->rank = rank;
    p->nranks = nranks;
    p->src = *src;
    p->dst = *dst;
    for (int r = 0; r < nranks; ++r)
    {
        p->src_boxes.push_back(to_box(src_boxes[r], nd));
        p->dst_boxes.push_back(to_box(dst_boxes[r], nd));
        for (int i = 0; i < nd; ++i)
            if (src_boxes[r].ext[i] < 0 || dst_boxes[r].ext[i] < 0 || src_boxes[r].off[i] < 0 || dst_boxes[r].off[i] < 0)
            {
                delete p;
                set_last_error("bad argument: negative box");
                return DCB_BAD_ARG;
            }
    }
    int32_t st = check_shard(src, p->src_boxes[rank], nd);
    if (st == DCB_OK)
        st = check_shard(dst, p->dst_boxes[rank], nd);
    if (st != DCB_OK)
    {
        delete p;
        return st;
    }
    // the window holds my destination block twice; a multiple of 4 floats so that
    // both parities start 16-byte aligned
    p->parity_floats = (p->dst_boxes[rank].volume() + 3) / 4 * 4;
    st = p->win.allocate(SHF_HEADER + (size_t) p->parity_floats * 2 * sizeof(float));
    if (st != DCB_OK)
    {
        delete p;
        return st;
    }
    p->peer_map.resize((size_t) nranks);
    *out = p;
    return DCB_OK;
}

int32_t dcb_shuffle_plan_destroy(dcb_shuffle_plan* p)
{
    if (!p)
        return DCB_OK;
    for (auto& m : p->peer_map)
        m.close();
    cudaFree(p->d_put);
    cudaFree(p->d_wait);
    p->win.release();
    delete p;
    return DCB_OK;
}

int32_t dcb_shuffle_plan_export(dcb_shuffle_plan* p, void* blob)
{
    DCB_REQUIRE(p && blob, "null argument");
    ShfBlob b;
    std::memset(&b, 0, sizeof(b));
    p->win.fill_blob(&b.win);
    b.rank = (uint32_t) p->rank;
    b.parity_floats = (uint64_t) p->parity_floats;
    std::memset(blob, 0, DCB_SHUFFLE_BLOB_BYTES);
    std::memcpy(blob, &b, sizeof(b));
    return DCB_OK;
}

int32_t dcb_shuffle_plan_connect(dcb_shuffle_plan* p, const void* blobs, int32_t nranks)
{
    DCB_REQUIRE(p && blobs, "null argument");
    DCB_REQUIRE(nranks == p->nranks, "blob count does not match the plan");
    const int nd = p->nd;
    long long ss[DCB_MAX_DIMS], ds[DCB_MAX_DIMS];
    real_strides(p->src, ss);
    real_strides(p->dst, ds);
    const Box& my_src = p->src_boxes[p->rank];
    const Box& my_dst = p->dst_boxes[p->rank];
    std::vector<ShfJob> put, wait;
    p->put_units = p->wait_units = 0;
    for (int r = 0; r < nranks; ++r)
    {
        Box x;
        // what I hold of rank r's destination block
        if (my_src.volume() > 0 && p->dst_boxes[r].volume() > 0 && intersect(my_src, p->dst_boxes[r], &x))
        {
            ShfBlob b;
            std::memcpy(&b, static_cast<const char*>(blobs) + (size_t) r * DCB_SHUFFLE_BLOB_BYTES, sizeof(b));
            DCB_REQUIRE((int) b.rank == r, "blob order does not match ranks");
            char* base = nullptr;
            if (r == p->rank)
                base = static_cast<char*>(p->win.base);
            else
            {
                const int32_t st = p->peer_map[r].open(b.win, p->win.device);
                if (st != DCB_OK)
                    return st;
                base = static_cast<char*>(p->peer_map[r].base);
            }
            DCB_REQUIRE((long long) b.parity_floats == (p->dst_boxes[r].volume() + 3) / 4 * 4,
                        "peer window does not match its destination block");
            ShfJob j;
            std::memset(&j, 0, sizeof(j));
            j.len = x.ext[0];
            j.rows = 1;
            j.a_off = j.b_off = 0;
            long long dense = 1; // strides of r's dense window
            for (int i = 0; i < DCB_MAX_DIMS; ++i)
            {
                const long long a_i = x.off[i] - my_src.off[i] + (i < nd ? p->src.overlap[i] : 0);
                const long long b_i = x.off[i] - p->dst_boxes[r].off[i];
                j.a_off += a_i * ss[i];
                j.b_off += b_i * dense;
                if (i >= 1)
                {
                    j.ext[i - 1] = x.ext[i];
                    j.a_stride[i - 1] = ss[i];
                    j.b_stride[i - 1] = dense;
                    j.rows *= x.ext[i];
                }
                dense *= p->dst_boxes[r].ext[i];
            }
            j.peer = reinterpret_cast<float*>(base + SHF_HEADER);
            j.parity_pitch = (long long) b.parity_floats;
            j.flag = reinterpret_cast<uint32_t*>(base) + p->rank; // my slot among r's flags
            add_jobs(j, &put, &p->put_units);
        }
        // what rank r holds of my destination block
        if (my_dst.volume() > 0 && p->src_boxes[r].volume() > 0 && intersect(p->src_boxes[r], my_dst, &x))
        {
            ShfJob j;
            std::memset(&j, 0, sizeof(j));
            j.len = x.ext[0];
            j.rows = 1;
            long long dense = 1;
            for (int i = 0; i < DCB_MAX_DIMS; ++i)
            {
                const long long a_i = x.off[i] - my_dst.off[i] + (i < nd ? p->dst.overlap[i] : 0);
                const long long b_i = x.off[i] - my_dst.off[i];
                j.a_off += a_i * ds[i];
                j.b_off += b_i * dense;
                if (i >= 1)
                {
                    j.ext[i - 1] = x.ext[i];
                    j.a_stride[i - 1] = ds[i];
                    j.b_stride[i - 1] = dense;
                    j.rows *= x.ext[i];
                }
                dense *= my_dst.ext[i];
            }
            j.peer = nullptr;
            j.flag = p->flags() + r;
            add_jobs(j, &wait, &p->wait_units);
        }
    }
    cudaFree(p->d_put);
    cudaFree(p->d_wait);
    p->d_put = p->d_wait = nullptr;
    for (int aligned = 0; aligned < 2; ++aligned)
    {
        auto pieces = [&](const ShfJob& j) { return shf_way(j.vec, j.len, aligned) == SHF_PIECE; };
        p->put_pieces[aligned] = std::any_of(put.begin(), put.end(), pieces);
        p->wait_pieces[aligned] = std::any_of(wait.begin(), wait.end(), pieces);
    }
    // (ranks that share a device share this process, or are not known to share it)
    double windows = 0;
    for (int r = 0; r < nranks; ++r)
    {
        ShfBlob b;
        std::memcpy(&b, static_cast<const char*>(blobs) + (size_t) r * DCB_SHUFFLE_BLOB_BYTES, sizeof(b));
        if (r == p->rank || (b.win.pid == (int32_t) getpid() && b.win.device == p->win.device))
            windows += 4.0 * (double) ((p->dst_boxes[r].volume() + 3) / 4 * 4);
    }
    int l2_bytes = 0;
    DCB_CUDA_TRY(cudaDeviceGetAttribute(&l2_bytes, cudaDevAttrL2CacheSize, p->win.device));
    p->from_the_end = shf_from_the_end(windows, l2_bytes);
    p->n_put = (int) put.size();
    p->n_wait = (int) wait.size();
    if (p->n_put)
    {
        DCB_CUDA_TRY(cudaMalloc(&p->d_put, put.size() * sizeof(ShfJob)));
        DCB_CUDA_TRY(cudaMemcpy(p->d_put, put.data(), put.size() * sizeof(ShfJob), cudaMemcpyHostToDevice));
    }
    if (p->n_wait)
    {
        DCB_CUDA_TRY(cudaMalloc(&p->d_wait, wait.size() * sizeof(ShfJob)));
        DCB_CUDA_TRY(cudaMemcpy(p->d_wait, wait.data(), wait.size() * sizeof(ShfJob), cudaMemcpyHostToDevice));
    }
    p->connected = true;
    return DCB_OK;
}

static unsigned shf_grid(long long units)
{
    const long long cap = (long long) num_sms() * 8;
    return (unsigned) (units < 1 ? 1 : (units > cap ? cap : units));
}

int32_t dcb_shuffle_put(dcb_shuffle_plan* p, const void* src, void* stream)
{
    DCB_REQUIRE(p, "null plan");
    if (!p->connected)
    {
        set_last_error("shuffle plan is not connected");
        return DCB_NOT_CONNECTED;
    }
    ++p->epoch;
    if (p->n_put == 0)
        return DCB_OK;
    DCB_REQUIRE(src, "null tensor");
    ShfArgs a;
    std::memset(&a, 0, sizeof(a));
    a.jobs = p->d_put;
    a.njobs = p->n_put;
    a.aligned = (reinterpret_cast<uintptr_t>(src) & 15) == 0;
    a.tensor = const_cast<float*>(static_cast<const float*>(src));
    a.parity = (int) (p->epoch & 1u);
    a.epoch = p->epoch;
    a.ticket = p->ticket();
    a.status = p->status();
    a.budget_ns = wait_budget_ns();
    (p->put_pieces[a.aligned] ? shuffle_kernel<true, true, false> : shuffle_kernel<true, false, false>)<<<shf_grid(p->put_units), SHF_THREADS, 0,
                                                                                        as_stream(stream)>>>(a);
    DCB_LAUNCH_CHECK();
    return DCB_OK;
}

int32_t dcb_shuffle_wait_unpack(dcb_shuffle_plan* p, void* dst, void* stream)
{
    DCB_REQUIRE(p, "null plan");
    if (!p->connected)
    {
        set_last_error("shuffle plan is not connected");
        return DCB_NOT_CONNECTED;
    }
    if (p->n_wait == 0)
        return DCB_OK;
    DCB_REQUIRE(dst, "null tensor");
    ShfArgs a;
    std::memset(&a, 0, sizeof(a));
    a.jobs = p->d_wait;
    a.njobs = p->n_wait;
    a.aligned = (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
    a.tensor = static_cast<float*>(dst);
    a.window = p->window() + (long long) (p->epoch & 1u) * p->parity_floats;
    a.epoch = p->epoch;
    a.ticket = p->ticket();
    a.status = p->status();
    a.budget_ns = wait_budget_ns();
    auto kernel = p->wait_pieces[a.aligned] ? shuffle_kernel<false, true, false>
                  : p->from_the_end        ? shuffle_kernel<false, false, true>
                                           : shuffle_kernel<false, false, false>;
    kernel<<<shf_grid(p->wait_units), SHF_THREADS, 0, as_stream(stream)>>>(a);
    DCB_LAUNCH_CHECK();
    return DCB_OK;
}

int32_t dcb_shuffle(dcb_shuffle_plan* p, const void* src, void* dst, void* stream)
{
    const int32_t st = dcb_shuffle_put(p, src, stream);
    if (st != DCB_OK)
        return st;
    return dcb_shuffle_wait_unpack(p, dst, stream);
}

int32_t dcb_shuffle_plan_status(dcb_shuffle_plan* p, void* stream)
{
    DCB_REQUIRE(p, "null plan");
    DCB_CUDA_TRY(cudaStreamSynchronize(as_stream(stream)));
    int st = 0;
    DCB_CUDA_TRY(cudaMemcpy(&st, p->status(), sizeof(int), cudaMemcpyDeviceToHost));
    if (st != 0)
    {
        const int zero = 0;
        DCB_CUDA_TRY(cudaMemcpy(p->status(), &zero, sizeof(int), cudaMemcpyHostToDevice));
    }
    return st;
}

} // extern "C"
