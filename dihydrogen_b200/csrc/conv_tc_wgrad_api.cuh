// Backward filter (conv_tc_wgrad.cuh): geometry and launch functions, one source
// file per stride along W (the kernels take long to compile).
#pragma once

#include "conv_simt.cuh"
#include "conv_tc_common.cuh"

namespace dcb
{

constexpr int WG_FLUSH = 4;  // warps 0..3: running sums, one per lane quadrant
constexpr int WG_CONV = 15;  // converter warps (20 warps in all leave 96 registers a thread)
constexpr int WG_ISSUE_WARP = WG_FLUSH + WG_CONV;
constexpr int WG_THREADS = (WG_FLUSH + WG_CONV + 1) * 32;
constexpr int WG_MAX_STAGES = 8;
constexpr int WG_MAX_TILES = 24;
constexpr int WG_CHAIN = 120; // updates of an accumulator: 2.5e-6 of the result on the longest sums (128^3)

struct WgTile
{
    uint32_t a16, b16; // first rows of the operands in a stage, 16-byte units
    uint32_t dcol, idesc;
};

struct WgGeom
{
    int n, c, k;
    int in[3], out[3], f[3], pad[3], stride[3];
    long long xs_n, xs_c, xs[3], ys_n, ys_c, ys[3];
    int cg, ncg, kwg, nkw, kdg, nkd, kg, kgp, nkg; // channels, taps kw, planes kd, filters per role and their groups
    int roles, parts;
    int ring;             // stages follow each other along D and keep the planes of x: see the kernel
    int A, X, B, PW, Q;   // input rows per tile, input and dy rows per stage, positions and cells of a row
    int r8, n8;           // matrix rows of an input row, of a dy row
    int xrows, yrows;     // matrix rows of a stage
    int lbo_x, lbo_y;     // bytes between cells of consecutive positions
    int stage_bytes, y_off, nstages;
    int ntiles, kd_a16, kd_cols; // tiles of one kd plane, distance between the planes' operands and accumulators
    int nclasses, class_lo[2], class_n[2], class_col[2]; // accumulator blocks: (a0 mod sh, b - a0 / sh)
    int nblocks;          // blocks per kd plane
    int sum_col;          // first column of the running sums
    int flush_stages;     // stages between flushes
    int hblocks, wchunks;
    int warps_x;          // converter warps that read x
    int items_x, items_y, cq, kq, qg; // warp items of a stage: channel and filter quadruples, cell groups of a row
    long long stages;     // per role
    // 16-byte loads: strides and bases allow them; x starts skip_x cells above a 16-byte boundary
    int vec_x, vec_y, skip_x;
    int so_tiles, so_items, so_bars, smem;
    WgTile tiles[WG_MAX_TILES];
};

// The dealing out for a forward geometry on `sms` multiprocessors; false where the
// kernel does not cover it.
bool wg_geom(const ConvGeom& cg, int math_mode, int sms, WgGeom* out);
// part[slice][role][filter gradient of the role] of the taps from rkw on; al: see
// the kernel's template parameter.
int32_t wg_launch_s1(const WgGeom& g, int al, int rkw, const float* x, const float* dy, float* part, int* status,
                     cudaStream_t stream);
int32_t wg_launch_s2(const WgGeom& g, int al, int rkw, const float* x, const float* dy, float* part, int* status,
                     cudaStream_t stream);

} // namespace dcb
