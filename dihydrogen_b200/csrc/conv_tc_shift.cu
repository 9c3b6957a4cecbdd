// Shift kernel, host side: filter image, device buffers, launches.
#include "conv_tc_shift_api.cuh"

#include "conv_plan_cache.cuh"
#include "conv_tc_encode.cuh"
#include "conv_tc_shift_plan.cuh"

#include <type_traits>

namespace dcb
{

namespace
{

__global__ void sh_pack_filter_kernel(const float* __restrict__ w, uint4* __restrict__ out,
                                      const ShPack* __restrict__ packs, const ShChunk* __restrict__ chunks,
                                      const int* __restrict__ codes, int kind, int parts, int total16, int cgroups,
                                      int cpg, int cin, int kout, int kcols, long long w_ko, long long w_ci,
                                      uint32_t rnd_add, uint32_t rnd_mask, float alpha, uint32_t* w_flag, uint32_t call)
{
    dependents_may_start();
    // the tables are the plan's: only the filter and the image have to wait
    const ShPack p = packs[blockIdx.y];
    const int kg = (int) blockIdx.z / cgroups, grp = (int) blockIdx.z % cgroups;
    uint4* o = out + (size_t) blockIdx.z * total16 + p.off16;
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = v < p.n * p.nchunks;
    const int c = v / p.n, col = v - c * p.n;
    ShChunk ck = {};
    int code = -1;
    if (on)
        ck = chunks[p.chunk0 + c], code = codes[p.code0 + col];
    wait_for_previous_kernel(w);
    if (!on)
        return;
    const int ko = kg * kcols + (code >> 16);
    const int ch0 = grp * cpg + ck.ch;
    const int CH = kind == 0 ? 4 : 8;
    const bool any = ck.part >= 0 && code >= 0 && ko < kout;
    const float* wp = w + ((long long) ko * w_ko + (long long) ch0 * w_ci + (code & 0xffff) + ck.kw);
    float f[8];
#pragma unroll
    for (int e = 0; e < 8; ++e)
        f[e] = any && e < CH && ch0 + e < cin && ck.ch + e < cpg ? alpha * wp[e * w_ci] : 0.f;
    float most = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e)
        most = fmaxf(most, fabsf(f[e]) <= 3.402823466e+38f ? 0.f : 1.f);
    if (most != 0.f)
        *w_flag = call;
    uint32_t r[8];
#pragma unroll
    for (int e = 0; e < 8; ++e)
    {
        if (kind == 0)
        {
            const uint32_t hi = round_operand(f[e], rnd_add, rnd_mask);
            r[e] = ck.part <= 0 ? hi : tf32_rna(f[e] - __uint_as_float(hi));
        }
        else if (parts == 1)
            r[e] = round_operand(f[e], rnd_add, 0xffffffffu);
        else
        {
#pragma unroll
            for (int s = 0; s < 2; ++s)
                if (s < ck.part)
                    f[e] -= __uint_as_float(__float_as_uint(f[e]) & 0xffff0000u);
            r[e] = __float_as_uint(f[e]);
        }
    }
    if (kind == 0)
        o[v] = make_uint4(r[0], r[1], r[2], r[3]);
    else
        o[v] = make_uint4(pack_hi16(r[0], r[1]), pack_hi16(r[2], r[3]), pack_hi16(r[4], r[5]), pack_hi16(r[6], r[7]));
}

// sums / sqsums[k] from the per epilogue warp partials of a launch, in order, in fp64.
constexpr int SH_FOLD_WARPS = 32;
__global__ void __launch_bounds__(SH_FOLD_WARPS * 32)
    sh_stats_fold_kernel(const float* __restrict__ part, int nparts, int nk, float* __restrict__ sums,
                         float* __restrict__ sqsums)
{
    __shared__ double sm[SH_FOLD_WARPS][32];
    const int t = threadIdx.x & 31, w = threadIdx.x >> 5;
    dependents_may_start();
    wait_for_previous_kernel(part);
    double acc = 0.0;
#pragma unroll 1
    for (int i = w; i < nparts; i += SH_FOLD_WARPS * 16)
    {
        // 16 loads in flight: the kernel is three trips to memory and nothing else
        float v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k)
            v[k] = i + k * SH_FOLD_WARPS < nparts ? part[(size_t) (i + k * SH_FOLD_WARPS) * 32 + t] : 0.f;
#pragma unroll
        for (int k = 0; k < 16; ++k)
            acc += (double) v[k];
    }
    sm[w][t] = acc;
    __syncthreads();
    if (w != 0)
        return;
    acc = 0.0;
#pragma unroll
    for (int i = 0; i < SH_FOLD_WARPS; ++i)
        acc += sm[i][t];
    if (t < 16)
    {
        if (t < nk)
            sums[t] = (float) acc;
    }
    else if (t - 16 < nk)
        sqsums[t - 16] = (float) acc;
}

} // namespace

struct ShPlan
{
    ShTables t;
    uint8_t* dev = nullptr; // one allocation: filter images, tables, packing tables, partial sums, status
    uint4* image = nullptr;
    uint8_t* tables = nullptr;
    ShPack* packs = nullptr;
    ShChunk* chunks = nullptr;
    int* codes = nullptr;
    float* stat_part = nullptr;
    uint32_t* w_flag = nullptr; // two: numbers of the last call whose filter, whose output had an element that is no number
    uint32_t call = 0;
    int max_image = 0;
};

bool sh_plan_create(const ConvGeom& g, bool transposed, int math_mode, ShPlan** out, int32_t* status)
{
    *out = nullptr;
    *status = DCB_OK;
    static PlanCache<std::pair<bool, ShTables>> cache;
    std::pair<bool, ShTables> found;
    cache.get(plan_key(g, transposed ? 1 : 0, math_mode), &found, [&]() {
        std::pair<bool, ShTables> r;
        r.first = ShBuilder(g, transposed, math_mode, num_sms()).build(&r.second);
        return r;
    });
    auto* p = new ShPlan();
    p->t = std::move(found.second);
    if (!found.first)
    {
        delete p;
        return false;
    }
    const ShTables& t = p->t;
    auto up = [](size_t v) { return (v + 255) / 256 * 256; };
    const size_t img = up((size_t) t.total16 * 16 * t.g.kgroups * t.g.cgroups), tab = up(t.blob.size()),
                 pk = up(t.packs.size() * sizeof(ShPack)), ck = up(t.chunks.size() * sizeof(ShChunk)),
                 cd = up(t.codes.size() * sizeof(int)),
                 sp = up(sh_has_stats(p) ? (size_t) num_sms() * SH_EPI * 32 * sizeof(float) : 0);
    std::vector<uint8_t> host(tab + pk + ck + cd, 0);
    std::memcpy(host.data(), t.blob.data(), t.blob.size());
    std::memcpy(host.data() + tab, t.packs.data(), t.packs.size() * sizeof(ShPack));
    std::memcpy(host.data() + tab + pk, t.chunks.data(), t.chunks.size() * sizeof(ShChunk));
    std::memcpy(host.data() + tab + pk + ck, t.codes.data(), t.codes.size() * sizeof(int));
    if (cudaMalloc(&p->dev, img + host.size() + sp + 2 * sizeof(uint32_t)) != cudaSuccess
        || cudaMemset(p->dev + img + host.size() + sp, 0, 2 * sizeof(uint32_t)) != cudaSuccess
        || cudaMemcpy(p->dev + img, host.data(), host.size(), cudaMemcpyHostToDevice) != cudaSuccess)
    {
        (void) cudaGetLastError();
        set_last_error("cudaMalloc of a convolution's tables failed");
        cudaFree(p->dev);
        delete p;
        *status = DCB_CUDA_ERROR;
        return false;
    }
    p->image = reinterpret_cast<uint4*>(p->dev);
    p->tables = p->dev + img;
    p->packs = reinterpret_cast<ShPack*>(p->tables + tab);
    p->chunks = reinterpret_cast<ShChunk*>(p->tables + tab + pk);
    p->codes = reinterpret_cast<int*>(p->tables + tab + pk + ck);
    p->stat_part = reinterpret_cast<float*>(p->tables + tab + pk + ck + cd);
    p->w_flag = reinterpret_cast<uint32_t*>(p->dev + img + host.size() + sp);
    for (const ShPack& k : t.packs)
        p->max_image = std::max(p->max_image, k.n * k.nchunks);
    *out = p;
    return true;
}

void sh_plan_destroy(ShPlan* p)
{
    if (!p)
        return;
    cudaFree(p->dev);
    delete p;
}

bool sh_has_stats(const ShPlan* p)
{
    const ShGeom& g = p->t.g;
    return g.kgroups == 1 && g.nb <= 16 && g.e_s * g.e_r * g.e_w == 1;
}

double sh_estimate(const ShPlan* p)
{
    return p->t.cost / 1900.0;
}

bool sh_bf16_split(const ShPlan* p)
{
    return p->t.parts == 3;
}

// The output as a 5-D tensor (W, R, S, filters, samples) whose box is what one
// epilogue warp stores: 32 positions of every filter of a group.
static bool sh_make_y_map(const ShGeom& g, float* y, CUtensorMap* map)
{
    EncodeTiledFn fn = encode_tiled_fn();
    // A bulk tensor store was seen to clip a row at the next 16-byte boundary,
    // not at the tensor's extent: rows of whole 16-byte pieces only.
    if (!fn || g.stage == 0 || (reinterpret_cast<uintptr_t>(y) & 15) != 0 || g.o_w % 4 != 0)
        return false;
    const cuuint64_t dims[5] = {(cuuint64_t) g.o_w, (cuuint64_t) g.o_r, (cuuint64_t) g.o_s, (cuuint64_t) g.kout,
                                (cuuint64_t) g.n};
    // a dimension of extent 1 may carry any stride; give it a valid one
    const long long sr = g.o_r > 1 ? g.ys_r : g.o_w, ss = g.o_s > 1 ? g.ys_s : sr * g.o_r;
    const long long sc = g.kout > 1 ? g.ys_c : ss * g.o_s, sn = g.n > 1 ? g.ys_n : sc * g.kout;
    const cuuint64_t strides[4] = {(cuuint64_t) sr * 4, (cuuint64_t) ss * 4, (cuuint64_t) sc * 4, (cuuint64_t) sn * 4};
    for (int i = 0; i < 4; ++i)
        if (strides[i] % 16 != 0 || strides[i] == 0)
            return false;
    const cuuint32_t box[5] = {32, 1, 1, (cuuint32_t) g.kcols, 1};
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, y, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
           == CUDA_SUCCESS;
}

int32_t sh_conv(ShPlan* p, float alpha, const float* x, const float* w, float beta, float* y, int* status,
                cudaStream_t stream, float* sums, float* sqsums)
{
    const ShTables& t = p->t;
    const ShGeom& g = t.g;
    const bool stats = sums != nullptr;
    if (stats && (beta != 0.f || !sh_has_stats(p)))
        return DCB_UNSUPPORTED;
    DCB_CUDA_TRY(launch_overlapped(sh_pack_filter_kernel,
                                   dim3((unsigned) ((p->max_image + 255) / 256), (unsigned) t.packs.size(),
                                        (unsigned) (g.kgroups * g.cgroups)),
                                   256, 0, stream, w, p->image, p->packs, p->chunks, p->codes, t.kind, t.parts, t.total16,
                                   g.cgroups, g.cpg, g.cin, g.kout, g.kcols, t.w_ko, t.w_ci, g.rnd_add, g.rnd_mask, alpha, p->w_flag, ++p->call));
    CUtensorMap ymap;
    std::memset(&ymap, 0, sizeof(ymap));
    const int use_ymap = beta == 0.f && sh_make_y_map(g, y, &ymap) ? 1 : 0;
    const unsigned grid = std::min<unsigned>((unsigned) num_sms(), g.units);
    const size_t smem = std::max<size_t>(t.smem, 120 * 1024); // one CTA per SM: it owns all of tensor memory
    ShExact exact = t.exact;
    exact.w_flag = p->w_flag;
    exact.out_flag = p->w_flag + 1;
    exact.call = p->call;
    exact.x = x;
    exact.w = w;
    exact.alpha = alpha;
    auto launch = [&](auto kernel, auto size) -> int32_t {
        const int32_t set = allow_dynamic_smem(reinterpret_cast<const void*>(kernel), 227 * 1024);
        if (set != DCB_OK)
            return set;
        ShConst<decltype(size)::value> ct;
        std::memcpy(&ct, t.issue.data(), t.issue.size());
        // starts beside the packing kernel: what it sets up does not depend on it
        DCB_CUDA_TRY(launch_overlapped(kernel, dim3(grid), SH_THREADS, smem, stream, g, exact, beta, ct, x, p->image, p->tables, y,
                                       status, p->stat_part, ymap, use_ymap));
        return DCB_OK;
    };
    auto dispatch = [&](auto wide, auto size) -> int32_t {
        constexpr bool W = decltype(wide)::value;
        constexpr int C = decltype(size)::value;
        auto with = [&](auto epilogue) -> int32_t {
            constexpr int E = decltype(epilogue)::value;
            if (t.kind == 0)
                return t.parts == 1 ? launch(sh_conv_kernel<0, 1, E, W, C>, size) : launch(sh_conv_kernel<0, 2, E, W, C>, size);
            return t.parts == 1 ? launch(sh_conv_kernel<1, 1, E, W, C>, size) : launch(sh_conv_kernel<1, 3, E, W, C>, size);
        };
        // (statistics are of plain outputs of 16 filters at most: never of blocks with two halves)
        return stats                ? with(std::integral_constant<int, SH_STATS>())
               : sh_shared_drain(g) ? with(std::integral_constant<int, SH_SHARED>())
                                    : with(std::integral_constant<int, SH_PLAIN>());
    };
    using Large = std::integral_constant<int, SH_CONST>;
    using Small = std::integral_constant<int, SH_CONST_SMALL>;
    const int32_t st = t.wide ? dispatch(std::true_type(), Large())
                              : (t.issue.size() > SH_CONST_SMALL ? dispatch(std::false_type(), Large())
                                                                 : dispatch(std::false_type(), Small()));
    if (st == DCB_OK && t.parts == 1 && beta == 0.f && g.st_s * g.st_r * g.st_w * g.e_s * g.e_r * g.e_w > 1)
        DCB_CUDA_TRY(launch_overlapped(stats ? sh_repair_kernel<true> : sh_repair_kernel<false>, dim3(grid), SH_THREADS, 0,
                                       stream, g, exact, y, p->stat_part));
    if (st != DCB_OK || !stats)
        return st;
    DCB_CUDA_TRY(launch_overlapped(sh_stats_fold_kernel, dim3(1), SH_FOLD_WARPS * 32, 0, stream, p->stat_part,
                                   (int) grid * SH_EPI, g.kout, sums, sqsums));
    return DCB_OK;
}

} // namespace dcb
