// tcgen05 sweep kernel (forward, few input channels) and backward filter, host
// side: geometry, tensor maps, launches.
#include "conv_tc.cuh"
#include "conv_plan_cache.cuh"
#include "conv_tc_encode.cuh"
#include "conv_tc_sweep.cuh"
#include "conv_tc_wgrad_api.cuh"

#include <cstdlib>
#include <type_traits>
#include <vector>

namespace dcb
{

namespace
{

size_t sw_smem_need(const SwGeom& g)
{
    return (size_t) (g.b_bytes + 127) / 128 * 128 + (size_t) g.raw_slots * g.raw_slot_bytes
           + (size_t) ((g.kr + 1) & ~1) * 4 + (size_t) (2 * g.a_slots + 64 + 2 * g.raw_slots + TC_GROUPS_MAX) * 8 + 64 + 128
           + (size_t) SW_EPI * 2 * SW_NBK * 32 * 4 + 1024;
}

// Geometry of the sweep kernel (filters with depth).  Needs bulk-copy
// compatible strides; the base address is checked per call.
bool sw_geom(const ConvGeom& cg, int math_mode, SwGeom* out)
{
    SwGeom g;
    std::memset(&g, 0, sizeof(g));
    for (int i = 0; i < 3; ++i)
    {
        if (cg.stride[i] != 1 || cg.dil[i] != 1)
            return false;
        g.in[i] = cg.in[i];
        g.out[i] = cg.out[i];
        g.f[i] = cg.f[i];
        g.pad[i] = cg.pad[i];
        g.xs[i] = cg.xs[i];
        g.ys[i] = cg.ys[i];
        if (g.pad[i] > g.f[i] - 1)
            return false;
    }
    g.n = cg.n;
    g.k = cg.k;
    g.xs_n = cg.xs_n;
    g.xs_c = cg.xs_c;
    g.ys_n = cg.ys_n;
    g.ys_c = cg.ys_c;
    if (g.f[0] < 2 || g.f[0] > 4 || g.k > SW_NBK)
        return false;
    // Its tiles are 128 outputs of a row; the shift kernel lays narrow rows, or parts of rows, side by
    // side.  Measured (4 -> 16 channels, 64 x 80 rows, with statistics, us, this kernel / shift kernel): rows
    // of 100 43.1 / 48.6, of 128 43.0 / 48.7, of 200 59.6 / 75.5; with whole rows only, rows of 56 40 / 31, of 32 22 / 18.
    if (2 * g.out[2] < (g.out[2] + TC_M - 1) / TC_M * TC_M)
        return false;
    g.split = (math_mode == DCB_MATH_TF32 || math_mode == DCB_MATH_BF16) ? 0 : 1;
    g.rnd_add = math_mode == DCB_MATH_BF16 ? 0x8000u : 0x1000u;
    g.rnd_mask = math_mode == DCB_MATH_BF16 ? 0xffff0000u : 0xffffe000u;
    // Three A slots of at most 53 k-rows each fit beside the accumulators.
    g.c = cg.c;
    if (3 * ((g.c * g.f[2] * (g.split ? 3 : 1) + 7) / 8 * 8) > 160)
        return false;
    if ((long long) cg.n * cg.out[0] * cg.out[1] * cg.out[2] == 0)
        return false;
    if (g.pad[2] > 4 || g.f[2] - 1 - g.pad[2] > 4)
        return false;
    if (!(cg.xs[1] % 4 == 0 && cg.xs[0] % 4 == 0 && cg.xs_c % 4 == 0 && cg.xs_n % 4 == 0))
        return false;
    g.ntot = g.f[1] * g.f[0] * SW_NBK;
    if (g.ntot > 256 || (g.f[0] * SW_NBK) % 16)
        return false;
    g.crows = g.c * g.f[2];
    g.kr = (g.crows * (g.split ? 2 : 1) + 7) / 8 * 8;
    g.ks1 = g.kr / 8;
    g.ksteps = g.ks1 + (g.split ? (g.crows + 7) / 8 : 0);
    g.kb = g.ksteps * 8;
    g.b_rot_bytes = g.kb * g.ntot * 4;
    g.b_bytes = g.f[0] * g.b_rot_bytes;
    // an issuer must own one of any fh consecutive rows (see the hand-off
    // notes in the kernel header): at most fh groups
    g.groups = g.f[1] < TC_GROUPS_MAX ? g.f[1] : TC_GROUPS_MAX;
    if (g.groups * g.kr > 160)
        return false;
    g.a_slots = g.groups;
    if (g.a_slots * g.kr > 256)
        return false;
    int th_max = ((int) TC_TMEM_COLS - g.a_slots * g.kr) / (g.f[0] * SW_NBK);
    if (th_max + g.f[1] - 1 > 32)
        th_max = 32 - g.f[1] + 1;
    if (th_max > g.out[1])
        th_max = g.out[1];
    if (th_max < 2)
        return false;
    // Rows per column (th) and segments along D (nseg) together decide how
    // evenly the units fill the SMs: take the pair with the fewest staged
    // rows on the busiest SM.  Fewer rows per column cost more halo rows,
    // more segments cost more spill steps; both are in the count.
    const int sms = num_sms();
    long long best_cost = -1;
    int best_th = th_max, best_ns = 1;
    for (int th = th_max; th >= 2 && th >= th_max - 3; --th)
    {
        const long long cols = (long long) g.n * ((g.out[2] + TC_M - 1) / TC_M) * ((g.out[1] + th - 1) / th);
        for (int ns = 1; ns <= g.out[0] && ns <= 64; ++ns)
        {
            const long long units = cols * ns;
            const long long waves = (units + sms - 1) / sms;
            const long long steps = (g.out[0] + ns - 1) / ns + 2 * (g.f[0] - 1);
            const long long cost = waves * steps * (th + g.f[1] - 1);
            if (best_cost < 0 || cost < best_cost)
            {
                best_cost = cost;
                best_th = th;
                best_ns = ns;
            }
        }
    }
    g.th = best_th;
    g.nseg = best_ns;
    g.rows = g.th + g.f[1] - 1;
    // Two A slots per group (and with them a second issuer per group in the plain
    // kernel) where the chosen column height leaves the tensor-memory columns for them:
    // the height is chosen first, by staged rows alone.
    if (2 * g.groups * g.kr <= 256
        && 2 * g.groups * g.kr + g.th * g.f[0] * SW_NBK <= (int) TC_TMEM_COLS)
        g.a_slots = 2 * g.groups;
    // chunks of about 17 KiB, evenly sized
    const int row_bytes = g.c * TC_RAW_W * 4;
    int rc_max = (17 * 1024 + 512) / row_bytes;
    rc_max = rc_max < 1 ? 1 : rc_max;
    g.chunks_pp = (g.rows + rc_max - 1) / rc_max;
    g.chunk_rows = (g.rows + g.chunks_pp - 1) / g.chunks_pp;
    g.raw_slot_bytes = (g.chunk_rows * row_bytes + 127) / 128 * 128;
    int slots = (72 * 1024) / g.raw_slot_bytes;
    slots = slots > 6 ? 6 : slots;
    if (slots < 2)
        return false;
    g.raw_slots = slots;
    // more epilogue warps need more staging buffers: a shallower ring pays for them
    while (g.raw_slots > 3 && sw_smem_need(g) > 200 * 1024)
        --g.raw_slots;
    if (sw_smem_need(g) > 200 * 1024)
        return false;
    g.tiles_w = (g.out[2] + TC_M - 1) / TC_M;
    g.tiles_h = (g.out[1] + g.th - 1) / g.th;
    g.units = (long long) g.n * g.tiles_w * g.tiles_h * g.nseg;
    if (g.units >= (1ll << 31))
        return false;
    *out = g;
    return true;
}

} // namespace

static size_t wg_part_floats(const WgGeom& g)
{
    return (size_t) g.nkw * g.roles * g.parts * g.kg * g.cg * g.kdg * g.f[1] * g.kwg;
}

struct TcPlan
{
    bool has_sw = false;
    SwGeom sw;
    float* sw_bimg = nullptr;
    float* stat_part = nullptr; // per epilogue warp partial sums of the fused statistics
    bool has_wg = false;
    WgGeom wg;
    float* wg_part = nullptr; // the CTAs' parts of the filter gradient
};

int32_t tc_plan_create(const ConvGeom& fwd, int math_mode, TcPlan** out)
{
    *out = nullptr;
    auto* p = new TcPlan();
    p->has_sw = sw_geom(fwd, math_mode, &p->sw);
    static PlanCache<std::pair<bool, WgGeom>> cache;
    std::pair<bool, WgGeom> found;
    cache.get(plan_key(fwd, 2, math_mode == DCB_MATH_FP32_SIMT), &found, [&]() {
        std::pair<bool, WgGeom> r;
        std::memset(&r.second, 0, sizeof(r.second));
        r.first = wg_geom(fwd, math_mode, num_sms(), &r.second);
        return r;
    });
    p->has_wg = found.first;
    p->wg = found.second;
    if (!p->has_sw && !p->has_wg)
    {
        delete p;
        return DCB_OK;
    }
    bool ok = true;
    if (p->has_sw)
        ok = cudaMalloc(&p->sw_bimg, p->sw.b_bytes) == cudaSuccess
             && cudaMalloc(&p->stat_part, (size_t) num_sms() * SW_EPI * 32 * sizeof(float)) == cudaSuccess;
    if (ok && p->has_wg)
        ok = cudaMalloc(&p->wg_part, wg_part_floats(p->wg) * sizeof(float)) == cudaSuccess;
    if (!ok)
    {
        (void) cudaGetLastError();
        set_last_error("cudaMalloc of a tensor-core plan failed");
        tc_plan_destroy(p);
        return DCB_CUDA_ERROR;
    }
    *out = p;
    return DCB_OK;
}

void tc_plan_destroy(TcPlan* p)
{
    if (!p)
        return;
    cudaFree(p->sw_bimg);
    cudaFree(p->stat_part);
    cudaFree(p->wg_part);
    delete p;
}

bool tc_has_sweep(const TcPlan* p)
{
    return p && p->has_sw;
}

bool tc_has_bwd_filter(const TcPlan* p)
{
    return p && p->has_wg;
}

// Floats between the 16-byte boundary at or below x and x.  A shard with halo cells
// along W is laid out so that its OWNED cells start on a 16-byte boundary (stores and
// the streaming kernels want that); its window, which starts with the halo cells, then
// does not.  A bulk copy can over-fetch but not start in between, so such a window is
// described from the boundary below it and the kernel skips the cells in front.  Those
// cells lie in the same allocation (allocations start 16-byte aligned) and are only read.
static inline int x_skip(const float* x)
{
    return (int) ((reinterpret_cast<uintptr_t>(x) & 15) / 4);
}

// Where a staged row starts relative to the first output of a tile (lx) and where tap 0
// sits in it (rx).  Aligned window: 4 cells of margin on the left for the padding.
// Skipped cells in front (only with pad 0): the row starts at the tile's first output.
template <class Geom>
static void tc_row_window(Geom& g, int skip)
{
    g.lx = skip ? 0 : -4;
    g.rx = skip ? skip : 4 - g.pad[2];
}

// can a window that starts `skip` floats above a 16-byte boundary be staged in rows of row_w cells?
static bool skip_ok(int skip, int pad_w, int fw, int tile_w, int row_w)
{
    if (skip == 0)
        return true;
    // cells left of the window are not zeros here, so nothing may read them as padding
    return pad_w == 0 && skip + fw - 1 + tile_w <= row_w;
}

// Descriptor of the input window as a 5-D tensor (W, H, D, C, N) whose box is
// chunk_rows raw rows of every channel.  Returns false when the window cannot be
// described (alignment), in which case the shift kernel runs.
static bool sw_make_x_map(const SwGeom& g, const float* x, CUtensorMap* map)
{
    EncodeTiledFn fn = encode_tiled_fn();
    const int skip = x_skip(x);
    if (!fn || (reinterpret_cast<uintptr_t>(x) & 3) != 0 || !skip_ok(skip, g.pad[2], g.f[2], TC_M, TC_RAW_W))
        return false;
    x -= skip;
    const cuuint64_t dims[5] = {(cuuint64_t) (g.in[2] + skip), (cuuint64_t) g.in[1], (cuuint64_t) g.in[0],
                                (cuuint64_t) g.c, (cuuint64_t) g.n};
    // a dimension of extent 1 may carry any stride; give it a valid one
    const long long s1 = g.xs[1], s0 = g.in[0] > 1 ? g.xs[0] : g.xs[1] * g.in[1];
    const cuuint64_t strides[4] = {(cuuint64_t) s1 * 4, (cuuint64_t) s0 * 4, (cuuint64_t) g.xs_c * 4,
                                   (cuuint64_t) (g.n > 1 ? g.xs_n : g.xs_c * g.c) * 4};
    for (int i = 0; i < 4; ++i)
        if (strides[i] % 16 != 0 || strides[i] == 0)
            return false;
    const cuuint32_t box[5] = {(cuuint32_t) TC_RAW_W, (cuuint32_t) g.chunk_rows, 1, (cuuint32_t) g.c, 1};
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, const_cast<float*>(x), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
           == CUDA_SUCCESS;
}

// Descriptor of the output as a 5-D tensor (W, H, D, K, N) whose box is 32
// outputs of every filter: what one epilogue warp stores per row.  Returns
// false when the output cannot be described (alignment); the kernel then
// stores from registers.
static bool sw_make_y_map(const SwGeom& g, float* y, CUtensorMap* map)
{
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn || (reinterpret_cast<uintptr_t>(y) & 15) != 0)
        return false;
    // A bulk tensor store was seen to clip a row at the next 16-byte boundary,
    // not at the tensor's extent: a row of 11 outputs inside a wider allocation
    // (a column range of a shard) had its 12th cell overwritten.  Rows whose
    // extent is not a multiple of 4 floats take the register stores.
    if (g.out[2] % 4 != 0)
        return false;
    const cuuint64_t dims[5] = {(cuuint64_t) g.out[2], (cuuint64_t) g.out[1], (cuuint64_t) g.out[0], (cuuint64_t) g.k,
                                (cuuint64_t) g.n};
    const long long s1 = g.out[1] > 1 ? g.ys[1] : g.out[2];
    const long long s0 = g.out[0] > 1 ? g.ys[0] : s1 * g.out[1];
    const long long sc = g.k > 1 ? g.ys_c : s0 * g.out[0];
    const long long sn = g.n > 1 ? g.ys_n : sc * g.k;
    const cuuint64_t strides[4] = {(cuuint64_t) s1 * 4, (cuuint64_t) s0 * 4, (cuuint64_t) sc * 4, (cuuint64_t) sn * 4};
    for (int i = 0; i < 4; ++i)
        if (strides[i] % 16 != 0 || strides[i] == 0)
            return false;
    const cuuint32_t box[5] = {32, 1, 1, (cuuint32_t) SW_NBK, 1};
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, y, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
           == CUDA_SUCCESS;
}

int32_t tc_sweep_fwd(TcPlan* p, float alpha, const float* x, const float* w, float* y, int* status, cudaStream_t stream,
                     float* sums, float* sqsums)
{
    if (!p || !p->has_sw)
        return DCB_UNSUPPORTED;
    SwGeom g = p->sw;
    CUtensorMap map, ymap;
    std::memset(&map, 0, sizeof(map));
    std::memset(&ymap, 0, sizeof(ymap));
    if (!sw_make_x_map(g, x, &map))
        return DCB_UNSUPPORTED;
    tc_row_window(g, x_skip(x));
    const int use_ymap = sw_make_y_map(g, y, &ymap) ? 1 : 0;
    const long long total = (long long) g.b_bytes / 4;
    DCB_CUDA_TRY(launch_overlapped(sw_pack_filter_kernel, dim3((unsigned) ((total + 255) / 256)), 256, 0, stream, w,
                                   p->sw_bimg, g));
    size_t smem = sw_smem_need(g);
    smem = smem < 120 * 1024 ? 120 * 1024 : smem; // one CTA per SM: it owns all of tensor memory
    long long grid = (long long) num_sms();
    if (grid > g.units)
        grid = g.units;
    const bool stats = sums != nullptr;
    // second issuers for the plain variant only
    const bool xiss = !stats && g.a_slots == 2 * g.groups;
    auto launch = [&](auto kernel, int xi) -> int32_t {
        const int32_t set = allow_dynamic_smem(reinterpret_cast<const void*>(kernel), 224 * 1024);
        if (set != DCB_OK)
            return set;
        DCB_CUDA_TRY(launch_overlapped(kernel, dim3((unsigned) grid), sw_threads(xi), smem, stream, g, alpha, p->sw_bimg, y,
                                       status, map, ymap, use_ymap, p->stat_part));
        return DCB_OK;
    };
    auto variant = [&](auto channels, auto split) -> int32_t {
        constexpr int C = decltype(channels)::value;
        constexpr bool S = decltype(split)::value;
        return stats ? launch(sw_conv_kernel<C, S, true, 0>, 0)
                     : (xiss ? launch(sw_conv_kernel<C, S, false, 1>, 1) : launch(sw_conv_kernel<C, S, false, 0>, 0));
    };
    auto channels = [&](auto split) -> int32_t {
        switch (g.f[2] == 3 && g.pad[2] <= 1 ? g.c : 0)
        {
        case 1: return variant(std::integral_constant<int, 1>(), split);
        case 2: return variant(std::integral_constant<int, 2>(), split);
        case 3: return variant(std::integral_constant<int, 3>(), split);
        case 4: return variant(std::integral_constant<int, 4>(), split);
        default: return variant(std::integral_constant<int, 0>(), std::true_type()); // (looks at g.split)
        }
    };
    const int32_t st = g.split ? channels(std::true_type()) : channels(std::false_type());
    if (st != DCB_OK || !stats)
        return st;
    DCB_CUDA_TRY(launch_overlapped(sw_stats_fold_kernel, dim3(1), SW_FOLD_WARPS * 32, 0, stream, p->stat_part,
                                   (int) grid * SW_EPI, g.k, sums, sqsums));
    return DCB_OK;
}

// One element of the filter gradient by FMAs over all positions, by a warp.  For sums that are
// no numbers: an infinity has no second part (inf - inf), and rows outside dy are multiplied as
// zeros, so that the parts may hold a NaN where there is a number or an infinity.
static __device__ __noinline__ float wg_exact(const WgGeom& g, const float* __restrict__ x, const float* __restrict__ dy, int e)
{
    const int taps = g.f[0] * g.f[1] * g.f[2], lane = threadIdx.x & 31;
    const int kw = e % g.f[2], kh = e / g.f[2] % g.f[1], kd = e / (g.f[2] * g.f[1]) % g.f[0], c = e / taps % g.c, k = e / taps / g.c;
    float acc = 0.f;
    for (int n = 0; n < g.n; ++n)
        for (int od = 0; od < g.out[0]; ++od)
        {
            const int id = od * g.stride[0] + kd - g.pad[0];
            if (id < 0 || id >= g.in[0])
                continue;
            for (int oh = 0; oh < g.out[1]; ++oh)
            {
                const int ih = oh * g.stride[1] + kh - g.pad[1];
                if (ih < 0 || ih >= g.in[1])
                    continue;
                const float* xp = x + (long long) n * g.xs_n + (long long) c * g.xs_c + (long long) id * g.xs[0] + (long long) ih * g.xs[1];
                const float* dp = dy + (long long) n * g.ys_n + (long long) k * g.ys_c + (long long) od * g.ys[0] + (long long) oh * g.ys[1];
                for (int ow = lane; ow < g.out[2]; ow += 32)
                {
                    const int iw = ow * g.stride[2] + kw - g.pad[2];
                    if (iw >= 0 && iw < g.in[2])
                        acc = fmaf(xp[iw], dp[ow], acc);
                }
            }
            if (__any_sync(0xffffffffu, acc != acc))
                return __int_as_float(0x7fc00000); // and stays that
        }
    for (int o = 16; o > 0; o >>= 1)
        acc += __shfl_xor_sync(0xffffffffu, acc, o);
    return acc;
}

// dw from the per-CTA parts: eight lanes per element, parts in order.
static __global__ void __launch_bounds__(256) wg_fold_kernel(const __grid_constant__ WgGeom g, const float* __restrict__ part,
                                                      const float* __restrict__ x, const float* __restrict__ dy, float alpha,
                                                      float beta, float* dw)
{
    const int taps = g.f[0] * g.f[1] * g.f[2];
    const int e = (int) (blockIdx.x * 32 + threadIdx.x / 8), sub = threadIdx.x & 7;
    const bool on = e < g.k * g.c * taps;
    double s = 0.0;
    wait_for_previous_kernel(part, x, dy);
    if (on)
    {
        const int kw = e % g.f[2], kh = e / g.f[2] % g.f[1], kd = e / (g.f[2] * g.f[1]) % g.f[0];
        const int c = e / taps % g.c, k = e / taps / g.c;
        const int role = (k / g.kg * g.nkd + kd / g.kdg) * g.ncg + c / g.cg;
        const int per = g.kg * g.cg * g.kdg * g.f[1] * g.kwg;
        const float* p = part + ((long long) (kw / g.kwg) * g.parts * g.roles + role) * per
                         + ((((long long) (k % g.kg) * g.cg + c % g.cg) * g.kdg + kd % g.kdg) * g.f[1] + kh) * g.kwg
                         + kw % g.kwg;
        const long long step = (long long) g.roles * per;
#pragma unroll 4
        for (int i = sub; i < g.parts; i += 8)
            s += (double) p[i * step];
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
        s += __shfl_xor_sync(0xffffffffu, s, o, 8);
    float sum = (float) s;
    const unsigned bad = __ballot_sync(0xffffffffu, on && sub == 0 && !(fabsf(sum) <= 3.402823466e+38f));
    if (bad != 0)
#pragma unroll 1
        for (int q = 0; q < 4; ++q)
            if (bad >> (8 * q) & 1)
            {
                const float v = wg_exact(g, x, dy, __shfl_sync(0xffffffffu, e, 8 * q));
                sum = (threadIdx.x & 31) / 8 == q ? v : sum;
            }
    if (on && sub == 0)
        dw[e] = alpha * sum + (beta != 0.f ? beta * dw[e] : 0.f);
}

int32_t tc_conv_bwd_filter(TcPlan* p, float alpha, const float* x, const float* dy, float beta, float* dw, int* status,
                           cudaStream_t stream)
{
    if (!p || !p->has_wg)
        return DCB_UNSUPPORTED;
    WgGeom g = p->wg;
    auto mult4 = [](long long a, long long b, long long c, long long d) { return ((a | b | c | d) & 3) == 0; };
    g.skip_x = x_skip(x);
    // (a piece that reaches past a row's last cell stays inside that cell's 16 bytes)
    g.vec_x = mult4(g.n > 1 ? g.xs_n : 0, g.c > 1 ? g.xs_c : 0, g.in[0] > 1 ? g.xs[0] : 0, g.in[1] > 1 ? g.xs[1] : 0);
    g.vec_y = mult4(g.n > 1 ? g.ys_n : 0, g.k > 1 ? g.ys_c : 0, g.out[0] > 1 ? g.ys[0] : 0, g.out[1] > 1 ? g.ys[1] : 0)
              && (reinterpret_cast<uintptr_t>(dy) & 15) == 0;
    const long long per_launch = (long long) wg_part_floats(g) / g.nkw;
    for (int i = 0; i < g.nkw; ++i)
    {
        const int rkw = i * g.kwg, al = g.vec_x ? (rkw - g.pad[2] + g.skip_x) & 3 : -1;
        const int32_t st = (g.stride[2] == 2 ? wg_launch_s2 : wg_launch_s1)(g, al, rkw, x, dy, p->wg_part + i * per_launch,
                                                                            status, stream);
        if (st != DCB_OK)
            return st;
    }
    const int total = g.k * g.c * g.f[0] * g.f[1] * g.f[2];
    DCB_CUDA_TRY(launch_overlapped(wg_fold_kernel, dim3((unsigned) ((total + 31) / 32)), 256, 0, stream, g, p->wg_part,
                                   x, dy, alpha, beta, dw));
    return DCB_OK;
}

} // namespace dcb
