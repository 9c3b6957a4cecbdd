"""Convolution kernels against the oracle and against outputs of the
reference's own ref::Backend (golden fixtures).  fp32: 1e-5 relative."""
import ctypes
import math
import os

import numpy as np
import pytest
import torch

import dihydrogen_b200 as dc
from dihydrogen_b200 import _abi
from oracle import oracle as O

import emu
import layers
from conftest import GOLDEN, conv_fixtures

pytestmark = pytest.mark.gpu

TOL = 1e-5
MODES = [_abi.MATH_FP32_SIMT, _abi.MATH_FP32]


def _nd(a: torch.Tensor) -> _abi.NdDesc:
    d = _abi.NdDesc()
    nsd = a.dim() - 2
    d.nsd = nsd
    d.n, d.c = a.shape[0], a.shape[1]
    d.sn, d.sc = a.stride(0), a.stride(1)
    for i in range(3):
        d.dims[i], d.strides[i] = 1, 0
    for i in range(nsd):
        d.dims[3 - nsd + i] = a.shape[2 + i]
        d.strides[3 - nsd + i] = a.stride(2 + i)
    return d


def _cd(K, C, f, pads, strides, dil, mode):
    nsd = len(f)
    cd = _abi.ConvDesc()
    cd.nsd, cd.k, cd.c, cd.groups, cd.math_mode = nsd, K, C, 1, mode
    for i in range(3):
        cd.filter[i], cd.pads[i], cd.strides[i], cd.dilations[i] = 1, 0, 1, 1
    for i in range(nsd):
        cd.filter[3 - nsd + i], cd.pads[3 - nsd + i] = f[i], pads[i]
        cd.strides[3 - nsd + i], cd.dilations[3 - nsd + i] = strides[i], dil[i]
    return cd


class Plan:
    def __init__(self, x, w, y, pads, strides, dil, mode):
        cd = _cd(w.shape[0], w.shape[1], list(w.shape[2:]), pads, strides, dil, mode)
        xd, yd = _nd(x), _nd(y)
        self.p = ctypes.c_void_p()
        _abi.call("dcb_conv_plan_create", ctypes.byref(cd), ctypes.byref(xd), ctypes.byref(yd), ctypes.byref(self.p))

    def __del__(self):
        _abi.lib().dcb_conv_plan_destroy(self.p)

    def fwd(self, alpha, x, w, beta, y):
        _abi.call("dcb_conv_fwd", self.p, alpha, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(w.data_ptr()), beta,
                  ctypes.c_void_p(y.data_ptr()), None)

    def bwd_data(self, alpha, w, dy, beta, dx):
        _abi.call("dcb_conv_bwd_data", self.p, alpha, ctypes.c_void_p(w.data_ptr()), ctypes.c_void_p(dy.data_ptr()),
                  beta, ctypes.c_void_p(dx.data_ptr()), None)

    def bwd_filter(self, alpha, x, dy, beta, dw):
        _abi.call("dcb_conv_bwd_filter", self.p, alpha, ctypes.c_void_p(x.data_ptr()),
                  ctypes.c_void_p(dy.data_ptr()), beta, ctypes.c_void_p(dw.data_ptr()), None)


def run_all(x, w, dy, pads, strides, dil, mode, alpha=1.0, beta=0.0, y0=None, dx0=None, dw0=None):
    xs, ws, dys = (torch.from_numpy(a).cuda() for a in (x, w, dy))
    y = torch.from_numpy(y0).cuda() if y0 is not None else torch.zeros(dy.shape, device="cuda")
    dx = torch.from_numpy(dx0).cuda() if dx0 is not None else torch.zeros(x.shape, device="cuda")
    dw = torch.from_numpy(dw0).cuda() if dw0 is not None else torch.zeros(w.shape, device="cuda")
    p = Plan(xs, ws, y, pads, strides, dil, mode)
    p.fwd(alpha, xs, ws, beta, y)
    p.bwd_data(alpha, ws, dys, beta, dx)
    p.bwd_filter(alpha, xs, dys, beta, dw)
    torch.cuda.synchronize()
    # a tensor-core kernel that gave up on one of its bounded waits says so here
    assert _abi.lib().dcb_conv_plan_status(p.p, None) == _abi.OK, "a conv kernel gave up on a bounded wait"
    return y.cpu().numpy(), dx.cpu().numpy(), dw.cpu().numpy()


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("fname", conv_fixtures())
def test_against_reference_backend_outputs(fname, mode):
    z = np.load(os.path.join(GOLDEN, fname))
    x, w, dy = z["x"], z["w"], z["dy"]
    f = w.shape[-1]
    p = (f - 1) // 2
    y, dx, dw = run_all(x, w, dy, [p, p], [1, 1], [1, 1], mode)
    # ref::Backend itself rounds in fp32 per step: allow 2e-5 against it
    emu.assert_close(y, z["y"], 2e-5, "y")
    emu.assert_close(dx, z["dx"], 2e-5, "dx")
    emu.assert_close(dw, z["dw"], 2e-5, "dw")


# N, C, K, spatial, filter, pads, strides, dilations
GEOMS = [
    (1, 4, 16, (12, 16, 40), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1)),     # cfg2 shape family
    (2, 3, 5, (7, 9, 33), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1)),        # ragged
    (1, 16, 32, (9, 10, 36), (3, 3, 3), (1, 1, 1), (2, 2, 2), (1, 1, 1)),     # cfg3 layer 2 (stride 2)
    (2, 8, 8, (20, 70), (5, 5), (2, 2), (1, 1), (1, 1)),                      # cfg4 family
    (1, 4, 6, (8, 9, 34), (3, 3, 3), (0, 0, 0), (1, 1, 1), (1, 1, 1)),        # no padding
    (1, 2, 3, (15, 31), (3, 3), (2, 2), (1, 1), (2, 2)),                      # dilation 2
    (1, 3, 4, (11, 12, 130), (1, 1, 1), (0, 0, 0), (1, 1, 1), (1, 1, 1)),     # 1x1x1
    (1, 4, 16, (6, 6, 260), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1)),      # wide rows, several W tiles
    (3, 5, 7, (9, 21), (3, 3), (1, 1), (2, 2), (1, 1)),                       # 2-D stride 2, odd extents
    (1, 4, 8, (6, 9, 36), (3, 2, 3), (1, 0, 1), (1, 1, 1), (1, 1, 1)),        # two filter rows: two converter groups
    (2, 3, 5, (5, 6, 40), (2, 1, 3), (1, 0, 1), (1, 1, 1), (1, 1, 1)),        # one filter row: one converter group
    (2, 3, 12, (7, 10, 132), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1)),     # backward data: 12 channels -> 3 filters
    (1, 4, 16, (9, 30, 64), (3, 3, 3), (0, 1, 1), (1, 1, 1), (1, 1, 1)),      # backward data: tall columns, no padding in D
    (2, 32, 32, (12, 140), (5, 5), (2, 2), (1, 1), (1, 1)),                   # cfg4 channels
    (1, 24, 40, (10, 70), (3, 3), (1, 1), (1, 1), (1, 1)),                    # ragged last filter group
    (1, 16, 32, (6, 8, 36), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1)),      # 3-D, 32 filters
    (1, 16, 16, (5, 7, 40), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1)),      # 3-D, 16 channels
    (1, 8, 20, (7, 12, 280), (3, 3, 3), (1, 1, 1), (2, 2, 2), (1, 1, 1)),     # stride 2, two W tiles (ragged), grouped backward filter
    (2, 4, 16, (9, 300), (3, 3), (1, 1), (1, 2), (1, 1)),                     # stride 2 along W only
    (1, 3, 5, (10, 264), (5, 5), (2, 2), (2, 2), (1, 1)),                     # 5x5 stride 2
    (1, 4, 32, (6, 9, 40), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1)),       # backward data over 32 channels: leading products apart from the corrections
]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("geom", GEOMS)
def test_against_oracle(geom, mode):
    N, C, K, sp, f, pads, strides, dil = geom
    rng = np.random.default_rng(hash(geom) % 2**32)
    x = rng.normal(0, 1, (N, C, *sp)).astype(np.float32)
    w = rng.normal(0, np.sqrt(2.0 / (C * np.prod(f))), (K, C, *f)).astype(np.float32)
    osp = [O.conv_out_extent(i, ff, p, s, d) for i, ff, p, s, d in zip(sp, f, pads, strides, dil)]
    dy = rng.normal(0, 1, (N, K, *osp)).astype(np.float32)
    y, dx, dw = run_all(x, w, dy, list(pads), list(strides), list(dil), mode)
    emu.assert_close(y, O.conv_fwd(x, w, list(pads), list(strides), list(dil)), TOL, "y")
    dx_ref = np.zeros_like(x)
    O.conv_bwd_data(w, dy, dx_ref, list(pads), list(strides), list(dil))
    emu.assert_close(dx, dx_ref, TOL, "dx")
    emu.assert_close(dw, O.conv_bwd_filter(x, dy, f, list(pads), list(strides), list(dil)), TOL, "dw")


@pytest.mark.parametrize("mode", MODES)
def test_alpha_beta_blend(mode):
    N, C, K, sp, f = 1, 4, 16, (6, 8, 36), (3, 3, 3)
    rng = np.random.default_rng(9)
    x = rng.normal(size=(N, C, *sp)).astype(np.float32)
    w = rng.normal(0, 0.1, (K, C, *f)).astype(np.float32)
    dy = rng.normal(size=(N, K, *sp)).astype(np.float32)
    y0 = rng.normal(size=dy.shape).astype(np.float32)
    dx0 = rng.normal(size=x.shape).astype(np.float32)
    dw0 = rng.normal(size=w.shape).astype(np.float32)
    y, dx, dw = run_all(x, w, dy, [1] * 3, [1] * 3, [1] * 3, mode, alpha=0.5, beta=2.0, y0=y0, dx0=dx0, dw0=dw0)
    emu.assert_close(y, O.conv_fwd(x, w, [1] * 3, [1] * 3, alpha=0.5, beta=2.0, y=y0.copy()), TOL, "y")
    emu.assert_close(dx, O.conv_bwd_data(w, dy, dx0.copy(), [1] * 3, [1] * 3, alpha=0.5, beta=2.0), TOL, "dx")
    emu.assert_close(dw, O.conv_bwd_filter(x, dy, f, [1] * 3, [1] * 3, alpha=0.5, beta=2.0, dw=dw0.copy()), TOL, "dw")


@pytest.mark.parametrize("mode", MODES)
def test_alpha_beta_blend_with_channel_groups(mode):
    """Only the first channel group may scale the old output by beta."""
    N, C, K, sp, f = 1, 32, 20, (9, 133), (5, 5)
    rng = np.random.default_rng(19)
    x = rng.normal(size=(N, C, *sp)).astype(np.float32)
    w = rng.normal(0, 0.05, (K, C, *f)).astype(np.float32)
    dy = rng.normal(size=(N, K, *sp)).astype(np.float32)
    y0 = rng.normal(size=dy.shape).astype(np.float32)
    dx0 = rng.normal(size=x.shape).astype(np.float32)
    dw0 = rng.normal(size=w.shape).astype(np.float32)
    y, dx, dw = run_all(x, w, dy, [2, 2], [1, 1], [1, 1], mode, alpha=0.5, beta=-1.5, y0=y0, dx0=dx0, dw0=dw0)
    emu.assert_close(y, 0.5 * O.conv_fwd(x, w, [2, 2], [1, 1], [1, 1]) - 1.5 * y0, TOL, "y")
    dx_ref = np.zeros_like(x)
    O.conv_bwd_data(w, dy, dx_ref, [2, 2], [1, 1], [1, 1])
    emu.assert_close(dx, 0.5 * dx_ref - 1.5 * dx0, TOL, "dx")
    emu.assert_close(dw, 0.5 * O.conv_bwd_filter(x, dy, f, [2, 2], [1, 1]) - 1.5 * dw0, TOL, "dw")


def test_plan_rejects_inconsistent_output_extent():
    x = torch.zeros(1, 2, 8, 8, device="cuda")
    w = torch.zeros(3, 2, 3, 3, device="cuda")
    y = torch.zeros(1, 3, 7, 8, device="cuda")
    with pytest.raises(_abi.DcbError) as e:
        Plan(x, w, y, [1, 1], [1, 1], [1, 1], _abi.MATH_FP32)
    assert e.value.status == _abi.BAD_ARG


def test_bias_forward_backward():
    rng = np.random.default_rng(2)
    y0 = rng.normal(size=(2, 5, 6, 7, 9)).astype(np.float32)
    b = rng.normal(size=5).astype(np.float32)
    y = torch.from_numpy(y0).cuda()
    bt = torch.from_numpy(b).cuda()
    yd = _nd(y)
    _abi.call("dcb_bias_fwd", 1.0, ctypes.c_void_p(bt.data_ptr()), 1.0, ctypes.byref(yd),
              ctypes.c_void_p(y.data_ptr()), None)
    emu.assert_close(y.cpu().numpy(), y0 + b.reshape(1, 5, 1, 1, 1), 1e-6, "bias fwd")
    db = torch.zeros(5, device="cuda")
    _abi.call("dcb_bias_bwd", 1.0, ctypes.byref(yd), ctypes.c_void_p(y.data_ptr()), 0.0,
              ctypes.c_void_p(db.data_ptr()), None)
    emu.assert_close(db.cpu().numpy(), y.cpu().numpy().astype(np.float64).sum(axis=(0, 2, 3, 4)), 1e-5, "bias bwd")


def test_forward_with_fused_statistics_matches_separate_pass():
    """dcb_conv_fwd_stats: same output as dcb_conv_fwd, and the per-filter sums
    the epilogue returns equal a statistics pass over that output."""
    N, C, K, sp, f = 2, 4, 16, (10, 23, 152), (3, 3, 3)
    rng = np.random.default_rng(31)
    x = torch.from_numpy(rng.normal(0.3, 1, (N, C, *sp)).astype(np.float32)).cuda()
    w = torch.from_numpy(rng.normal(0, 0.1, (K, C, *f)).astype(np.float32)).cuda()
    y0 = torch.zeros(N, K, *sp, device="cuda")
    y1 = torch.full((N, K, *sp), 7.0, device="cuda")
    p = Plan(x, w, y0, [1] * 3, [1] * 3, [1] * 3, _abi.MATH_FP32)
    p.fwd(1.0, x, w, 0.0, y0)
    sums = torch.zeros(K, device="cuda")
    sq = torch.zeros(K, device="cuda")
    st = _abi.lib().dcb_conv_fwd_stats(p.p, 1.0, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(w.data_ptr()),
                                       ctypes.c_void_p(y1.data_ptr()), ctypes.c_void_p(sums.data_ptr()),
                                       ctypes.c_void_p(sq.data_ptr()), None)
    assert st == _abi.OK, st
    torch.cuda.synchronize()
    assert _abi.lib().dcb_conv_plan_status(p.p, None) == _abi.OK
    emu.assert_close(y1.cpu().numpy(), y0.cpu().numpy(), 2e-6, "y with statistics")
    ref = y0.double()
    emu.assert_close(sums.cpu().numpy(), ref.sum(dim=(0, 2, 3, 4)).cpu().numpy(), 1e-5, "sums")
    emu.assert_close(sq.cpu().numpy(), (ref * ref).sum(dim=(0, 2, 3, 4)).cpu().numpy(), 1e-5, "sqsums")


def test_fused_statistics_unsupported_for_2d():
    x = torch.zeros(1, 4, 16, 32, device="cuda")
    w = torch.zeros(8, 4, 3, 3, device="cuda")
    y = torch.zeros(1, 8, 16, 32, device="cuda")
    p = Plan(x, w, y, [1, 1], [1, 1], [1, 1], _abi.MATH_FP32)
    s = torch.zeros(8, device="cuda")
    st = _abi.lib().dcb_conv_fwd_stats(p.p, 1.0, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(w.data_ptr()),
                                       ctypes.c_void_p(y.data_ptr()), ctypes.c_void_p(s.data_ptr()),
                                       ctypes.c_void_p(s.data_ptr()), None)
    assert st == _abi.UNSUPPORTED


def test_tensor_core_kernels_are_the_ones_running():
    """For the bench layer's shape family all three passes resolve to tcgen05
    kernels (more channels: several launches on channel groups); a filter with
    more taps than tensor-memory lanes (> 128) keeps the fp32 kernel for the
    backward filter."""
    x = torch.zeros(1, 4, 8, 16, 128, device="cuda")
    w = torch.zeros(16, 4, 3, 3, 3, device="cuda")
    y = torch.zeros(1, 16, 8, 16, 128, device="cuda")
    p = Plan(x, w, y, [1] * 3, [1] * 3, [1] * 3, _abi.MATH_FP32)
    assert [_abi.lib().dcb_conv_plan_kernel_kind(p.p, i) for i in range(3)] == [1, 1, 1]
    x2 = torch.zeros(1, 8, 8, 16, 128, device="cuda")
    w2 = torch.zeros(16, 8, 3, 3, 3, device="cuda")
    p2 = Plan(x2, w2, y, [1] * 3, [1] * 3, [1] * 3, _abi.MATH_FP32)
    assert _abi.lib().dcb_conv_plan_kernel_kind(p2.p, 2) == 1
    x3 = torch.zeros(1, 2, 8, 16, 128, device="cuda")
    w3 = torch.zeros(16, 2, 5, 5, 7, device="cuda")
    p3 = Plan(x3, w3, y, [2, 2, 3], [1] * 3, [1] * 3, _abi.MATH_FP32)
    assert _abi.lib().dcb_conv_plan_kernel_kind(p3.p, 2) == 0


def test_backward_filter_tensor_core_ragged_tiles_and_batch():
    """Several W tiles with a ragged last one, N > 1, alpha / beta blend."""
    N, C, K, sp, f = 2, 4, 13, (5, 7, 268), (3, 3, 3)
    rng = np.random.default_rng(77)
    x = rng.normal(size=(N, C, *sp)).astype(np.float32)
    w = rng.normal(0, 0.1, (K, C, *f)).astype(np.float32)
    dy = rng.normal(size=(N, K, *sp)).astype(np.float32)
    dw0 = rng.normal(size=w.shape).astype(np.float32)
    _, _, dw = run_all(x, w, dy, [1] * 3, [1] * 3, [1] * 3, _abi.MATH_FP32, alpha=0.5, beta=2.0,
                       y0=np.zeros(dy.shape, np.float32), dx0=np.zeros(x.shape, np.float32), dw0=dw0)
    emu.assert_close(dw, O.conv_bwd_filter(x, dy, f, [1] * 3, [1] * 3, alpha=0.5, beta=2.0, dw=dw0.copy()), TOL, "dw")


@pytest.mark.parametrize("mode", MODES)
def test_backward_filter_full_shard_against_fp64_sums(mode):
    """The 256^3 shard of the benchmark: every filter gradient is a sum over
    16.7 M voxels, where an accumulator that truncates instead of rounding shows
    (4e-4 with one tensor-memory chain for the whole run).  Sampled taps are
    recomputed as fp64 dot products and must agree within the fp32 contract."""
    D = 256
    gen = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(1, 4, D, 256, 256, device="cuda", generator=gen)
    dy = torch.randn(1, 16, D, 256, 256, device="cuda", generator=gen)
    dy += 0.5  # a mean, so that sums do not hide a bias behind cancellation
    x += 0.25
    w = torch.zeros(16, 4, 3, 3, 3, device="cuda")
    dw = torch.zeros_like(w)
    p = Plan(x, w, dy, [1] * 3, [1] * 3, [1] * 3, mode)
    p.bwd_filter(1.0, x, dy, 0.0, dw)
    torch.cuda.synchronize()
    assert _abi.lib().dcb_conv_plan_status(p.p, None) == _abi.OK
    dyd = dy[0].double()
    got, ref = [], []
    for c, (td, th, tw) in [(0, (0, 0, 0)), (1, (1, 1, 1)), (2, (2, 2, 2)), (3, (0, 2, 1)), (1, (2, 0, 1)), (2, (1, 2, 0))]:
        # dw[k][c][t] = sum_o dy[k][o] * x[c][o + t - 1]
        xs = torch.zeros(D, 256, 256, device="cuda", dtype=torch.float64)
        sl_o, sl_i = [], []
        for t, n in ((td, D), (th, 256), (tw, 256)):
            lo, hi = max(0, 1 - t), min(n, n + 1 - t)
            sl_o.append(slice(lo, hi))
            sl_i.append(slice(lo + t - 1, hi + t - 1))
        xs[tuple(sl_o)] = x[0, c][tuple(sl_i)].double()
        ref.append((dyd * xs).sum(dim=(1, 2, 3)))
        got.append(dw[:, c, td, th, tw].double())
        del xs
    got, ref = torch.stack(got), torch.stack(ref)
    err = ((got - ref).abs() / (ref.abs() + ref.pow(2).mean().sqrt())).max().item()
    assert err <= TOL, err


def test_forward_with_statistics_full_shard():
    """The benchmark's 256^3 shard: the fused per-filter sums against fp64 sums
    of the output, and the output on a sampled block against an fp64 convolution."""
    D = 256
    gen = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn(1, 4, D, 256, 256, device="cuda", generator=gen) + 0.3
    w = torch.randn(16, 4, 3, 3, 3, device="cuda", generator=gen) * 0.14
    y = torch.zeros(1, 16, D, 256, 256, device="cuda")
    p = Plan(x, w, y, [1] * 3, [1] * 3, [1] * 3, _abi.MATH_FP32)
    sums, sq = torch.zeros(16, device="cuda"), torch.zeros(16, device="cuda")
    st = _abi.lib().dcb_conv_fwd_stats(p.p, 1.0, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(w.data_ptr()),
                                       ctypes.c_void_p(y.data_ptr()), ctypes.c_void_p(sums.data_ptr()),
                                       ctypes.c_void_p(sq.data_ptr()), None)
    assert st == _abi.OK, st
    torch.cuda.synchronize()
    assert _abi.lib().dcb_conv_plan_status(p.p, None) == _abi.OK
    s64, q64 = torch.zeros(16, dtype=torch.float64, device="cuda"), torch.zeros(16, dtype=torch.float64, device="cuda")
    for d0 in range(0, D, 32):
        blk = y[0, :, d0:d0 + 32].double()
        s64 += blk.sum(dim=(1, 2, 3))
        q64 += (blk * blk).sum(dim=(1, 2, 3))
    emu.assert_close(sums.cpu().numpy(), s64.cpu().numpy(), TOL, "sums")
    emu.assert_close(sq.cpu().numpy(), q64.cpu().numpy(), TOL, "sqsums")
    # a block that touches three faces of the shard and its far corner
    for sl in ((slice(0, 6), slice(0, 40), slice(0, 256)), (slice(D - 6, D), slice(216, 256), slice(0, 256))):
        lo = [max(0, s.start - 1) for s in sl]
        hi = [min(n, s.stop + 1) for s, n in zip(sl, (D, 256, 256))]
        xb = x[:, :, lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]].double()
        pad = []
        for s, l, h, n in reversed(list(zip(sl, lo, hi, (D, 256, 256)))):
            pad += [1 - (s.start - l), 1 - (h - s.stop)]
        ref = torch.nn.functional.conv3d(torch.nn.functional.pad(xb, pad), w.double())
        emu.assert_close(y[:, :, sl[0], sl[1], sl[2]].cpu().numpy(), ref.cpu().numpy(), TOL, "y block")


@pytest.mark.parametrize("W,pad", [(30, 1), (33, 1), (130, 1), (30, 0), (35, 0)])
def test_rows_padded_to_a_pitch_with_odd_extents(W, pad):
    """x, y (and dy, dx) live in allocations whose rows are padded to a pitch
    of 4 floats while the row EXTENT is not a multiple of 4: the bulk-copy fed
    kernels take them (strides are 16-byte multiples), so a row's last cells,
    the zero padding beyond them and the stores at the row's end are exactly
    what an off-by-a-granule tensor map would get wrong.  The padding cells
    are poisoned with NaN on the way in and must be untouched on the way out."""
    rng = np.random.default_rng(W)
    N, C, K, D, H = 1, 4, 16, 6, 9
    Wo = W + 2 * pad - 2
    Do, Ho = D + 2 * pad - 2, H + 2 * pad - 2
    x = rng.normal(size=(N, C, D, H, W)).astype(np.float32)
    w = rng.normal(0, 0.2, (K, C, 3, 3, 3)).astype(np.float32)
    dy = rng.normal(size=(N, K, Do, Ho, Wo)).astype(np.float32)

    def pitched(a):
        p = -(-a.shape[-1] // 4) * 4
        st = torch.full(a.shape[:-1] + (p,), float("nan"), device="cuda")
        v = st[..., :a.shape[-1]]
        v.copy_(torch.from_numpy(a))
        return st, v

    xs, xv = pitched(x)
    ys, yv = pitched(np.zeros(dy.shape, np.float32))
    dys, dyv = pitched(dy)
    dxs, dxv = pitched(np.zeros(x.shape, np.float32))
    wt = torch.from_numpy(w).cuda()
    dw = torch.zeros_like(wt)
    p = Plan(xv, wt, yv, [pad] * 3, [1] * 3, [1] * 3, _abi.MATH_FP32)
    assert [_abi.lib().dcb_conv_plan_kernel_kind(p.p, i) for i in range(3)] == [1, 1, 1]
    p.fwd(1.0, xv, wt, 0.0, yv)
    p.bwd_data(1.0, wt, dyv, 0.0, dxv)
    p.bwd_filter(1.0, xv, dyv, 0.0, dw)
    torch.cuda.synchronize()
    assert _abi.lib().dcb_conv_plan_status(p.p, None) == _abi.OK
    pads = [pad] * 3
    emu.assert_close(yv.cpu().numpy(), O.conv_fwd(x, w, pads, [1] * 3), TOL, "y")
    dx_ref = np.zeros_like(x)
    O.conv_bwd_data(w, dy, dx_ref, pads, [1] * 3)
    emu.assert_close(dxv.cpu().numpy(), dx_ref, TOL, "dx")
    emu.assert_close(dw.cpu().numpy(), O.conv_bwd_filter(x, dy, (3, 3, 3), pads, [1] * 3), TOL, "dw")
    for st, ext in ((ys, Wo), (dxs, W)):
        if st.shape[-1] > ext:
            assert bool(torch.isnan(st[..., ext:]).all()), "a store went past the end of a row"


def _round_bf16(a):
    """fp32 -> bf16, ties away from zero, as the kernels' integer rounding does."""
    b = a.astype(np.float32).view(np.uint32)
    return ((b + np.uint32(0x8000)) & np.uint32(0xFFFF0000)).view(np.float32)


@pytest.mark.parametrize("mode", [_abi.MATH_BF16, _abi.MATH_TF32])
@pytest.mark.parametrize("shape", [
    (1, 4, 16, (20, 23, 140), (3, 3, 3)),     # the bench layer's family: sweep kernel, shift kernel backward
    (2, 16, 8, (40, 70), (3, 3)),             # 2-D
    (1, 12, 16, (9, 17, 33), (3, 3, 3)),      # channel groups
])
def test_reduced_precision_modes_equal_the_rounded_operands_product(shape, mode):
    """DCB_MATH_BF16 / DCB_MATH_TF32: operands rounded to bf16 / TF32 on their way
    into the tensor cores, products exact, fp32 accumulation.  So forward and
    backward data must equal the fp64 convolution of the ROUNDED inputs and
    filters within the fp32 contract; the error against the unrounded operands
    is the rounding's (2^-9 / 2^-11 relative per operand).  Backward filter keeps
    fp32 quality in every mode."""
    N, C, K, sp, f = shape
    rng = np.random.default_rng(sum(sp) + mode)
    nsd = len(sp)
    pads = [1] * nsd
    x = rng.normal(size=(N, C) + tuple(sp)).astype(np.float32)
    w = rng.normal(0, 0.2, (K, C) + tuple(f)).astype(np.float32)
    dy = rng.normal(size=(N, K) + tuple(sp)).astype(np.float32)
    if mode == _abi.MATH_BF16:
        rnd = _round_bf16
    else:
        rnd = lambda a: ((a.view(np.uint32) + np.uint32(0x1000)) & np.uint32(0xFFFFE000)).view(np.float32)
    y, dx, dw = run_all(x, w, dy, pads, [1] * nsd, [1] * nsd, mode)
    emu.assert_close(y, O.conv_fwd(rnd(x), rnd(w), pads, [1] * nsd), TOL, "y")
    dx_ref = np.zeros_like(x)
    O.conv_bwd_data(rnd(w), rnd(dy), dx_ref, pads, [1] * nsd)
    emu.assert_close(dx, dx_ref, TOL, "dx")
    emu.assert_close(dw, O.conv_bwd_filter(x, dy, tuple(f), pads, [1] * nsd), TOL, "dw")
    # and the rounding is really there: against the unrounded product the bf16 result is ~1e-3 off
    full = O.conv_fwd(x, w, pads, [1] * nsd)
    err = np.abs(y - full).max() / np.abs(full).max()
    assert (1e-4 < err < 2e-2) if mode == _abi.MATH_BF16 else (1e-5 < err < 5e-3), err


@pytest.mark.parametrize("lead", [1, 2, 3])
@pytest.mark.parametrize("Wl", [32, 64, 35])
def test_window_that_starts_above_a_16_byte_boundary(lead, Wl):
    """The layout of a shard with halo cells along W: rows padded to a pitch,
    the OWNED cells of a row on a 16-byte boundary, so the halo-extended window
    starts `lead` floats above one (3 with one halo cell).  Forward and backward filter read such a
    window (no padding along W: the halo stands in for it) and write / read the
    owned cells; backward data reads the halo-extended dy and writes dx's owned
    cells (padding f - 1 in the descriptor's terms).  The tensor-core kernels
    must take all three (the bulk copies fetch from the boundary below the
    window and skip the cells in front), meet the 1e-5 contract and leave the
    lead and tail cells of every row alone."""
    rng = np.random.default_rng(100 * lead + Wl)
    N, C, K, D, H = 1, 4, 16, 5, 9
    We = Wl + 2

    def shard(a, off):
        pitch = -(-(off + a.shape[-1]) // 4) * 4
        st = torch.full(a.shape[:-1] + (pitch,), float("nan"), device="cuda")
        v = st[..., off:off + a.shape[-1]]
        v.copy_(torch.from_numpy(a))
        return st, v

    w = rng.normal(0, 0.2, (K, C, 3, 3, 3)).astype(np.float32)
    wt = torch.from_numpy(w).cuda()
    # forward and backward filter: x window of Wl + 2 cells `lead` floats into the row, y / dy
    # the Wl owned cells on a boundary
    x = rng.normal(size=(N, C, D, H, We)).astype(np.float32)
    dy = rng.normal(size=(N, K, D, H, Wl)).astype(np.float32)
    xs, xv = shard(x, lead)
    ys, yv = shard(np.zeros(dy.shape, np.float32), 4)
    dys, dyv = shard(dy, 4)
    assert xv.data_ptr() % 16 == 4 * lead and yv.data_ptr() % 16 == 0
    dw = torch.zeros_like(wt)
    pads = [1, 1, 0]
    p = Plan(xv, wt, yv, pads, [1] * 3, [1] * 3, _abi.MATH_FP32)
    assert _abi.lib().dcb_conv_plan_kernel_variant(p.p, 0) == 3
    p.fwd(1.0, xv, wt, 0.0, yv)
    p.bwd_filter(1.0, xv, dyv, 0.0, dw)
    torch.cuda.synchronize()
    assert _abi.lib().dcb_conv_plan_status(p.p, None) == _abi.OK
    emu.assert_close(yv.cpu().numpy(), O.conv_fwd(x, w, pads, [1] * 3), TOL, "y")
    emu.assert_close(dw.cpu().numpy(), O.conv_bwd_filter(x, dy, (3, 3, 3), pads, [1] * 3), TOL, "dw")
    assert bool(torch.isnan(ys[..., :4]).all()) and bool(torch.isnan(ys[..., 4 + Wl:]).all())
    # backward data: dy window with its halo, dx the owned cells
    dye = rng.normal(size=(N, K, D, H, We)).astype(np.float32)
    des, dev = shard(dye, lead)
    dxs, dxv = shard(np.zeros((N, C, D, H, Wl), np.float32), 4)
    pads_b = [1, 1, 2]
    pb = Plan(dxv, wt, dev, pads_b, [1] * 3, [1] * 3, _abi.MATH_FP32)
    pb.bwd_data(1.0, wt, dev, 0.0, dxv)
    torch.cuda.synchronize()
    assert _abi.lib().dcb_conv_plan_status(pb.p, None) == _abi.OK
    dx_ref = np.zeros((N, C, D, H, Wl), np.float32)
    O.conv_bwd_data(w, dye, dx_ref, pads_b, [1] * 3)
    emu.assert_close(dxv.cpu().numpy(), dx_ref, TOL, "dx")
    assert bool(torch.isnan(dxs[..., :4]).all()) and bool(torch.isnan(dxs[..., 4 + Wl:]).all())


@pytest.mark.parametrize("lead", [1, 3])
def test_stride_2_backward_filter_on_a_window_above_a_16_byte_boundary(lead):
    """The stride-2 layer of a W-partitioned tensor: x is read with its halo from
    `lead` floats above a 16-byte boundary (no padding along W), dy's owned cells
    sit on one.  The tcgen05 backward filter must take it (two half windows per
    unit, every second cell) and meet the contract."""
    rng = np.random.default_rng(lead)
    N, C, K, Wl = 1, 4, 16, 70
    D, H = 9, 11
    We = 2 * Wl + 1
    Do, Ho = (D + 2 - 3) // 2 + 1, (H + 2 - 3) // 2 + 1

    def shard(a, off):
        pitch = -(-(off + a.shape[-1]) // 4) * 4
        st = torch.full(a.shape[:-1] + (pitch,), float("nan"), device="cuda")
        v = st[..., off:off + a.shape[-1]]
        v.copy_(torch.from_numpy(a))
        return st, v

    x = rng.normal(size=(N, C, D, H, We)).astype(np.float32)
    w = rng.normal(0, 0.2, (K, C, 3, 3, 3)).astype(np.float32)
    dy = rng.normal(size=(N, K, Do, Ho, Wl)).astype(np.float32)
    xs, xv = shard(x, lead)
    dys, dyv = shard(dy, 4)
    wt = torch.from_numpy(w).cuda()
    dw = torch.zeros_like(wt)
    pads, strides = [1, 1, 0], [2, 2, 2]
    p = Plan(xv, wt, dyv, pads, strides, [1] * 3, _abi.MATH_FP32)
    assert _abi.lib().dcb_conv_plan_kernel_variant(p.p, 2) == 5
    p.bwd_filter(1.0, xv, dyv, 0.0, dw)
    torch.cuda.synchronize()
    assert _abi.lib().dcb_conv_plan_status(p.p, None) == _abi.OK
    emu.assert_close(dw.cpu().numpy(), O.conv_bwd_filter(x, dy, (3, 3, 3), pads, strides), TOL, "dw")


def test_backward_data_full_shard_16_channels_against_fp64():
    """Backward data of the benchmark layer on its 256^3 shard: dy has 16
    channels, six products of three bf16 parts; the leading ones have an accumulator
    set of their own (a single truncating chain of 180 updates sat on the 1e-5 bound).  dy carries a mean so that a truncation bias cannot
    hide behind cancellation; sampled blocks of dx (a corner, an edge, the
    interior) are recomputed in fp64."""
    import torch.nn.functional as F

    D = 256
    gen = torch.Generator(device="cuda").manual_seed(13)
    dy = torch.randn(1, 16, D, 256, 256, device="cuda", generator=gen) + 0.5
    w = torch.randn(16, 4, 3, 3, 3, device="cuda", generator=gen) * 0.14 + 0.02
    dx = torch.full((1, 4, D, 256, 256), float("nan"), device="cuda")
    p = Plan(dx, w, dy, [1] * 3, [1] * 3, [1] * 3, _abi.MATH_FP32)
    assert _abi.lib().dcb_conv_plan_kernel_variant(p.p, 1) == 4, "expected the shift kernel on bf16 parts"
    for rep in range(3):  # the order in which the issuers' instructions land varies from run to run
        p.bwd_data(1.0, w, dy, 0.0, dx)
        torch.cuda.synchronize()
        assert _abi.lib().dcb_conv_plan_status(p.p, None) == _abi.OK
        assert not bool(torch.isnan(dx).any())
        worst = 0.0
        B = 12
        for o0 in ((0, 0, 0), (100, 0, 117), (244, 244, 244), (31, 200, 64)):
            lo = [max(0, o - 2) for o in o0]
            hi = [min(256, o + B + 2) for o in o0]
            blk = dy[0, :, lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]].double()
            full = F.conv_transpose3d(blk[None], w.double(), padding=1)[0]
            sl = tuple(slice(o - l, o - l + B) for o, l in zip(o0, lo))
            ref = full[(slice(None),) + sl]
            got = dx[0, :, o0[0]:o0[0] + B, o0[1]:o0[1] + B, o0[2]:o0[2] + B].double()
            worst = max(worst, ((got - ref).abs() / (ref.abs() + ref.pow(2).mean().sqrt())).max().item())
        assert worst <= TOL, (rep, worst)


@pytest.mark.parametrize("geom", [
    # N, C, K, spatial, filter, stride: edges of the shift kernel's tiles and tables
    (1, 8, 8, (5, 6, 9), (3, 3, 3), 1),        # six sub-columns side by side in the 128 lanes
    (1, 8, 8, (5, 6, 127), (3, 3, 3), 1),      # one cell short of a tile
    (1, 8, 8, (5, 6, 129), (3, 3, 3), 1),      # one cell over: two tiles
    (3, 9, 17, (4, 5, 31), (3, 3, 3), 1),      # a cell of one channel, 17 filters in 20 columns
    (1, 32, 32, (9, 34, 40), (3, 3, 3), 1),    # filter images streamed per plane, channel groups
    (2, 7, 33, (6, 7, 65), (3, 3, 3), 2),      # stride 2, filters in groups, odd extents
    (1, 31, 31, (13, 131), (5, 5), 2),         # 2-D 5 x 5 stride 2
    (2, 1, 4, (40, 17), (3, 3), 1),            # one channel, 2-D
    (1, 6, 5, (4, 4, 4), (3, 3, 3), 2),        # smallest
    (1, 1, 4, (900, 150), (3, 3), 1),          # few filters: blocks narrower than an instruction's 16 columns, many planes
    (1, 8, 4, (40, 60, 132), (3, 3, 3), 2),    # the same where a plane adds to some of the live slots only
    (1, 5, 24, (90, 84), (5, 5), 2),           # blocks of one and a half times 16 columns
    (2, 4, 4, (40, 17), (3, 3), 1),            # the layers of one channel above with products enough for this kernel
    (1, 16, 4, (900, 150), (3, 3), 1, [1, 0]),  # 4 filters: forward here, backward data on CUDA cores
    (1, 4, 16, (900, 150), (3, 3), 1, [0, 1]),  # the other way round
])
def test_shift_kernel_tile_and_table_edges(geom):
    N, C, K, sp, f, s = geom[:6]
    rng = np.random.default_rng(sum(sp) + C)
    nsd, pads, strides = len(sp), [(e - 1) // 2 for e in f], [s] * len(sp)
    x = rng.normal(0, 1, (N, C, *sp)).astype(np.float32)
    w = rng.normal(0, np.sqrt(2.0 / (C * np.prod(f))), (K, C, *f)).astype(np.float32)
    dy = rng.normal(0, 1, (N, K, *[O.conv_out_extent(i, ff, p, s, 1) for i, ff, p in zip(sp, f, pads)])).astype(np.float32)
    y0 = rng.normal(size=dy.shape).astype(np.float32)
    dx0 = rng.normal(size=x.shape).astype(np.float32)
    p = Plan(*(torch.from_numpy(a).cuda() for a in (x, w, dy)), pads, strides, [1] * nsd, _abi.MATH_FP32)
    kinds = [_abi.lib().dcb_conv_plan_kernel_kind(p.p, i) for i in (0, 1)]
    want = geom[6] if len(geom) > 6 else [1, 1]
    assert kinds == want or (C == 1 and nsd == 2), "one channel may take the CUDA cores, the others are here for the shift kernel"
    y, dx, _ = run_all(x, w, dy, pads, strides, [1] * nsd, _abi.MATH_FP32, alpha=0.5, beta=-1.0, y0=y0, dx0=dx0,
                       dw0=np.zeros_like(w))
    emu.assert_close(y, 0.5 * O.conv_fwd(x, w, pads, strides) - y0, TOL, "y")
    dx_ref = np.zeros_like(x)
    O.conv_bwd_data(w, dy, dx_ref, pads, strides)
    emu.assert_close(dx, 0.5 * dx_ref - dx0, TOL, "dx")


# strides that differ: an epilogue that fetches beyond its accumulators, after a kernel that left NaNs there
@pytest.mark.parametrize("mode", [_abi.MATH_FP32, _abi.MATH_BF16])
@pytest.mark.parametrize("channels,f,strides", [
    (4, 3, (2, 1, 1)), (4, 3, (1, 1, 2)), (3, 3, (2, 1, 2)), (4, 3, (1, 2, 1)), (8, 2, (1, 1, 2)), (4, 2, (1, 2, 2)),
    (5, 3, (2, 2, 1)),
])
def test_shift_kernel_strides_that_differ(channels, f, strides, mode):
    rng = np.random.default_rng(channels + f)
    sp, pads = (9, 18, 70), [(f - 1) // 2] * 3
    x = rng.normal(0, 1, (2, channels, *sp)).astype(np.float32)
    w = rng.normal(0, np.sqrt(2.0 / (channels * f ** 3)), (16, channels, f, f, f)).astype(np.float32)
    dy = rng.normal(0, 1, (2, 16, *[O.conv_out_extent(i, f, p, s, 1) for i, p, s in zip(sp, pads, strides)])).astype(np.float32)
    if mode == _abi.MATH_BF16:
        w, dy = _round_bf16(w), _round_bf16(dy)
    g = [torch.from_numpy(a).cuda() for a in (x, w, dy)]
    p = Plan(*g, pads, list(strides), [1] * 3, mode)
    assert _abi.lib().dcb_conv_plan_kernel_kind(p.p, 1) == 1, "expected the shift kernel"
    p.bwd_filter(1.0, g[0], torch.full_like(g[2], float("nan")), 0.0, torch.zeros_like(g[1]))
    dx = torch.full_like(g[0], float("nan"))
    p.bwd_data(1.0, g[1], g[2], 0.0, dx)
    dx_ref = np.zeros_like(x)
    O.conv_bwd_data(w, dy, dx_ref, pads, list(strides))
    emu.assert_close(dx.cpu().numpy(), dx_ref, TOL, "dx")


# the issuers' tables as an argument of 1 KB and of 8 KB
@pytest.mark.parametrize("geom", [
    (1, 4, 4, (9, 12, 40), (3, 3, 3), 1),
    (1, 16, 16, (12, 14, 40), (5, 5, 5), 1),
    (1, 4, 4, (16, 16, 16), (7, 7, 7), 1),
])
def test_shift_kernel_short_and_long_tables(geom):
    test_shift_kernel_tile_and_table_edges(geom)


@pytest.mark.parametrize("geom", [
    # N, C, K, spatial, filter, stride: edges of the backward filter's stages and roles
    (1, 4, 16, (5, 7, 32), (3, 3, 3), 1),      # one stage wide, rows left over
    (2, 3, 5, (3, 4, 33), (3, 3, 3), 1),       # rows no vector load can read, filters padded to 8
    (1, 33, 9, (9, 40), (3, 3), 1),            # channels in roles
    (1, 20, 40, (6, 6, 24), (3, 3, 3), 1),     # channels, planes kd and filters in roles
    (1, 32, 32, (21, 70), (5, 5), 1),          # five taps along W
    (1, 31, 7, (15, 67), (5, 5), 2),           # stride 2 with five taps
    (2, 2, 3, (11, 18), (2, 2), 2),            # two taps
    (1, 2, 3, (12, 36), (7, 7), 1),            # more taps than one launch takes
    (4, 1, 4, (200, 130), (3, 3), 1),          # long sums: running sums used
    (1, 4, 16, (37, 29, 70), (3, 3, 3), 1),    # walks along D that begin and end inside a column
    (2, 4, 16, (4, 101, 128), (3, 3, 3), 1),   # walks shorter than the ring of planes
    (1, 5, 7, (66, 50, 41), (2, 3, 3), 1),     # two planes kd, rows no vector load can read
])
def test_backward_filter_stage_and_role_edges(geom):
    N, C, K, sp, f, s = geom
    rng = np.random.default_rng(sum(sp) + K)
    nsd, pads, strides = len(sp), [(e - 1) // 2 for e in f], [s] * len(sp)
    x = rng.normal(0.2, 1, (N, C, *sp)).astype(np.float32)
    w = np.zeros((K, C, *f), np.float32)
    dy = rng.normal(0.1, 1, (N, K, *[O.conv_out_extent(i, ff, p, s, 1) for i, ff, p in zip(sp, f, pads)])).astype(np.float32)
    xs, ws, dys = (torch.from_numpy(a).cuda() for a in (x, w, dy))
    dw = torch.from_numpy(rng.normal(size=w.shape).astype(np.float32)).cuda()
    dw0 = dw.cpu().numpy()
    p = Plan(xs, ws, dys, pads, strides, [1] * nsd, _abi.MATH_FP32)
    assert _abi.lib().dcb_conv_plan_kernel_kind(p.p, 2) == 1
    p.bwd_filter(0.5, xs, dys, -2.0, dw)
    torch.cuda.synchronize()
    assert _abi.lib().dcb_conv_plan_status(p.p, None) == _abi.OK
    emu.assert_close(dw.cpu().numpy(), 0.5 * O.conv_bwd_filter(x, dy, f, pads, strides) - 2.0 * dw0, TOL, "dw")


def _relative_errors(N, C, K, sp, f, s, mode):
    """2-norm errors of y and dx against fp64; everything has a mean, so that the
    tensor pipe's truncation cannot hide behind cancellation."""
    import torch.nn.functional as F

    gen = torch.Generator(device="cuda").manual_seed(3)
    pads, osp = [(e - 1) // 2 for e in f], [O.conv_out_extent(i, e, (e - 1) // 2, s, 1) for i, e in zip(sp, f)]
    x = torch.randn(N, C, *sp, device="cuda", generator=gen) + 0.5
    w = torch.randn(K, C, *f, device="cuda", generator=gen) * (2.0 / (C * math.prod(f))) ** 0.5 + 0.02
    dy = torch.randn(N, K, *osp, device="cuda", generator=gen) + 0.3
    y, dx = torch.empty_like(dy), torch.empty_like(x)
    p = Plan(x, w, y, pads, [s] * len(sp), [1] * len(sp), mode)
    p.fwd(1.0, x, w, 0.0, y)
    p.bwd_data(1.0, w, dy, 0.0, dx)
    torch.cuda.synchronize()
    assert _abi.lib().dcb_conv_plan_status(p.p, None) == _abi.OK
    with torch.backends.cudnn.flags(enabled=False):
        xr = x.double().requires_grad_()
        yr = (F.conv3d if len(sp) == 3 else F.conv2d)(xr, w.double(), stride=s, padding=pads)
        yr.backward(dy.double())
    return [((a.double() - b).norm() / b.norm()).item() for a, b in ((y, yr.detach()), (dx, xr.grad))]


@pytest.mark.parametrize("geom", [
    (1, 128, 32, (8, 16, 32), (3, 3, 3)), (1, 256, 16, (8, 16, 32), (3, 3, 3)), (2, 128, 32, (28, 56), (5, 5)),
    (2, 32, 32, (32, 64), (11, 11)), (1, 16, 16, (9, 16, 32), (7, 7, 7)),
])
def test_wide_layers_do_not_accumulate_in_one_chain(geom):
    """A chain is at most 96 updates, each of which loses half a unit in the last
    place of a sum that has reached half its value on average: 96 * 2^-25 of the
    result, and as much again for the rounding of the sums."""
    N, C, K, sp, f = geom
    assert max(_relative_errors(N, C, K, sp, f, 1, _abi.MATH_FP32)) <= 96 * 2.0 ** -25


@pytest.mark.parametrize("geom", [
    (1, 16, 32, (24, 26, 70), (3, 3, 3), 2), (2, 64, 128, (28, 56), (3, 3), 2), (2, 3, 64, (56, 112), (7, 7), 2),
    (1, 32, 32, (16, 20, 67), (3, 3, 3), 1), (2, 32, 32, (48, 131), (5, 5), 2), (1, 4, 16, (24, 40, 67), (3, 3, 3), 2),
])
def test_strided_and_wide_layers_are_as_exact_as_fp32_fma(geom):
    """... whose error grows with the square root of the number of terms; 2^-22 for
    what does not depend on it (the split, the sum of the accumulators)."""
    got = _relative_errors(*geom, _abi.MATH_FP32)
    fma = _relative_errors(*geom, _abi.MATH_FP32_SIMT)
    assert all(a <= 1.25 * b + 2.0 ** -22 for a, b in zip(got, fma)), (got, fma)


@pytest.mark.parametrize("sp", [(5, 7, 132), (5, 7, 45)])
@pytest.mark.parametrize("channel_stride", [2 ** 28 + 64, 2 ** 30 + 64])
def test_channels_far_apart(channel_stride, sp):
    """Channels that lie further apart than 32-bit byte offsets reach, as in volumes of
    2^28 cells and more; the shorter rows are not the sweep kernel's."""
    N, C, K = 1, 4, 4
    rng = np.random.default_rng(5)
    x = rng.normal(size=(N, C, *sp)).astype(np.float32)
    w = rng.normal(0, 0.2, (K, C, 3, 3, 3)).astype(np.float32)
    dy = rng.normal(size=(N, K, *sp)).astype(np.float32)
    store = torch.empty(3 * channel_stride + sp[0] * sp[1] * sp[2], device="cuda")

    def far(a):
        v = store.as_strided(a.shape, (4 * channel_stride, channel_stride, sp[1] * sp[2], sp[2], 1))
        v.copy_(torch.from_numpy(a))
        return v

    wt, xf = torch.from_numpy(w).cuda(), far(x)
    y = torch.zeros(dy.shape, device="cuda")
    p = Plan(xf, wt, y, [1] * 3, [1] * 3, [1] * 3, _abi.MATH_FP32)
    assert _abi.lib().dcb_conv_plan_kernel_kind(p.p, 0) == 1
    p.fwd(1.0, xf, wt, 0.0, y)
    emu.assert_close(y.cpu().numpy(), O.conv_fwd(x, w, [1] * 3, [1] * 3), TOL, "y")
    dyn, dw = torch.from_numpy(dy).cuda(), torch.zeros_like(wt)
    p.bwd_filter(1.0, xf, dyn, 0.0, dw)
    emu.assert_close(dw.cpu().numpy(), O.conv_bwd_filter(x, dy, (3, 3, 3), [1] * 3, [1] * 3), TOL, "dw")
    dyf = far(dy)
    dx = torch.zeros(x.shape, device="cuda")
    pb = Plan(dx, wt, dyf, [1] * 3, [1] * 3, [1] * 3, _abi.MATH_FP32)
    assert _abi.lib().dcb_conv_plan_kernel_kind(pb.p, 1) == 1
    pb.bwd_data(1.0, wt, dyf, 0.0, dx)
    dx_ref = np.zeros_like(x)
    O.conv_bwd_data(w, dy, dx_ref, [1] * 3, [1] * 3)
    emu.assert_close(dx.cpu().numpy(), dx_ref, TOL, "dx")
    assert _abi.lib().dcb_conv_plan_status(p.p, None) == _abi.lib().dcb_conv_plan_status(pb.p, None) == _abi.OK


@pytest.mark.parametrize("geom", [
    (1, 16, 16, (24, 40, 67), (3, 3, 3), 1), (2, 8, 24, (33, 41, 51), (3, 3, 3), 1), (2, 31, 17, (96, 131), (5, 5), 1),
    (1, 16, 32, (24, 40, 64), (3, 3, 3), 2), (2, 32, 32, (95, 131), (5, 5), 2), (1, 8, 24, (24, 40, 150), (3, 3, 3), 2),
])
def test_backward_filter_of_strided_and_unaligned_layers_is_as_exact_as_fp32_fma(geom):
    """... to half as much again, and 2^-21 for what does not depend on the number of
    positions (shortest chain between flushes: 16 updates of 2^-25 of the sum, the parts)."""
    import torch.nn.functional as F

    N, C, K, sp, f, s = geom
    gen = torch.Generator(device="cuda").manual_seed(4)
    pads, osp = [(e - 1) // 2 for e in f], [O.conv_out_extent(i, e, (e - 1) // 2, s, 1) for i, e in zip(sp, f)]
    x = torch.randn(N, C, *sp, device="cuda", generator=gen)
    x = torch.where(x < 0, 0.01 * x, x)
    dy = 1e-2 * torch.randn(N, K, *osp, device="cuda", generator=gen)
    w = torch.zeros(K, C, *f, device="cuda")
    with torch.backends.cudnn.flags(enabled=False):
        wr = w.double().requires_grad_()
        (F.conv3d if len(sp) == 3 else F.conv2d)(x.double(), wr, stride=s, padding=pads).backward(dy.double())
    errors = []
    for mode in (_abi.MATH_FP32, _abi.MATH_FP32_SIMT):
        p = Plan(x, w, dy, pads, [s] * len(sp), [1] * len(sp), mode)
        assert _abi.lib().dcb_conv_plan_kernel_kind(p.p, 2) == (mode == _abi.MATH_FP32)
        dw = torch.zeros_like(w)
        p.bwd_filter(1.0, x, dy, 0.0, dw)
        torch.cuda.synchronize()
        errors.append(((dw.double() - wr.grad).norm() / wr.grad.norm()).item())
    assert errors[0] <= 1.5 * errors[1] + 2.0 ** -21, errors


@pytest.mark.parametrize("geom", [
    # N, C, K, spatial, filter, stride, kernels of forward and backward data: either side of the rule
    (2, 1, 4, (512, 512), (3, 3), 1, (0, 0)), (2, 4, 8, (512, 512), (3, 3), 1, (0, 1)), (2, 4, 16, (512, 512), (3, 3), 1, (1, 1)),
    (2, 1, 4, (95, 131), (3, 3), 2, (0, 1)), (1, 8, 4, (64, 127, 128), (3, 3, 3), 2, (1, 0)), (1, 1, 16, (33, 64, 65), (3, 3, 3), 2, (0, 1)),
])
def test_layers_of_few_products_on_either_kernel(geom):
    N, C, K, sp, f, s, kinds = geom
    rng = np.random.default_rng(C + K)
    pads, strides = [1] * len(sp), [s] * len(sp)
    x = rng.normal(0, 1, (N, C, *sp)).astype(np.float32)
    w = rng.normal(0, np.sqrt(2.0 / (C * np.prod(f))), (K, C, *f)).astype(np.float32)
    dy = rng.normal(0, 1, (N, K, *[O.conv_out_extent(i, 3, 1, s, 1) for i in sp])).astype(np.float32)
    xs = torch.from_numpy(x).cuda()
    p = Plan(xs, torch.from_numpy(w).cuda(), torch.from_numpy(dy).cuda(), pads, strides, [1] * len(sp), _abi.MATH_FP32)
    assert tuple(_abi.lib().dcb_conv_plan_kernel_kind(p.p, i) for i in (0, 1)) == kinds
    y, dx, _ = run_all(x, w, dy, pads, strides, [1] * len(sp), _abi.MATH_FP32)
    emu.assert_close(y, O.conv_fwd(x, w, pads, strides), TOL, "y")
    dx_ref = np.zeros_like(x)
    O.conv_bwd_data(w, dy, dx_ref, pads, strides)
    emu.assert_close(dx, dx_ref, TOL, "dx")


NAN_ALL_ONES = np.uint32(0x7FFFFFFF).view(np.float32)  # what CUDA's arithmetic returns
NON_FINITE_GEOMS = [
    (1, 4, 16, (6, 9, 140), (3, 3, 3), 1),   # sweep kernel
    (1, 2, 8, (6, 9, 132), (3, 3, 3), 1),    # ... with fewer channels
    (1, 4, 16, (6, 9, 33), (3, 3, 3), 1),    # shift kernel, TF32 cells
    (1, 16, 16, (12, 37), (3, 3), 1),        # ... bf16 cells
    (2, 8, 16, (7, 9, 20), (3, 3, 3), 2),
    (1, 12, 20, (17, 30), (5, 5), 2),
]


@pytest.mark.parametrize("mode", [_abi.MATH_FP32, _abi.MATH_TF32, _abi.MATH_BF16])
@pytest.mark.parametrize("geom", NON_FINITE_GEOMS + [
    (1, 1, 8, (6, 9, 132), (3, 3, 3), 1), (1, 5, 16, (6, 9, 132), (3, 3, 3), 1),  # sweep kernel, the second with its general converter
])
def test_what_is_not_a_number_stays_that(geom, mode):
    """In every mode, in the input, the filter and the gradient."""
    N, C, K, sp, f, s = geom
    rng = np.random.default_rng(8)
    pads, strides, dil = [(e - 1) // 2 for e in f], [s] * len(sp), [1] * len(sp)
    x = rng.normal(size=(N, C, *sp)).astype(np.float32)
    w = rng.normal(size=(K, C, *f)).astype(np.float32)
    dy = rng.normal(size=(N, K, *[O.conv_out_extent(i, e, (e - 1) // 2, s, 1) for i, e in zip(sp, f)])).astype(np.float32)
    xn, wn, dyn = x.copy(), w.copy(), dy.copy()
    xn[(0, C - 1) + tuple(e // 2 for e in sp)] = dyn[(0, K - 1) + tuple(e // 2 for e in dy.shape[2:])] = NAN_ALL_ONES
    wn[(K - 1, 0) + tuple(e // 2 for e in f)] = NAN_ALL_ONES
    seen_y = O.conv_fwd(np.isnan(xn).astype(np.float32), np.ones_like(w), pads, strides) > 0
    seen_dx = np.zeros_like(x)
    O.conv_bwd_data(np.ones_like(w), np.isnan(dyn).astype(np.float32), seen_dx, pads, strides)
    y, dx, dw = run_all(xn, w, dyn, pads, strides, dil, mode)
    assert np.isnan(y[seen_y]).all() and np.isnan(dx[seen_dx > 0]).all()
    # (the gradient's NaN reaches all of its filter, the input's every tap that sees it)
    assert np.isnan(dw[K - 1]).all() and np.isnan(dw[:, C - 1]).any(axis=tuple(range(1, 1 + len(f)))).all()
    assert not np.isnan(dw[:K - 1, :C - 1]).any()
    y, dx, _ = run_all(x, wn, dy, pads, strides, dil, mode)
    assert np.isnan(y[:, K - 1]).any() and not np.isnan(y[:, :K - 1]).any()
    assert np.isnan(dx[:, 0]).any() and not np.isnan(dx[:, 1:]).any()


@pytest.mark.parametrize("value", [np.float32(np.inf), NAN_ALL_ONES])
@pytest.mark.parametrize("mode", [_abi.MATH_FP32, _abi.MATH_TF32, _abi.MATH_BF16])
@pytest.mark.parametrize("geom", NON_FINITE_GEOMS[2:] + [
    (1, 4, 4, (8, 9, 64), (3, 3, 3), 2),     # backward data: cells of four columns drained together
    (1, 8, 16, (20, 64), (3, 3), 1),         # bulk stores
    (1, 16, 24, (5, 6, 40), (3, 3, 3), 1),
    (1, 4, 8, (9, 33), (1, 1), 2),           # one tap: its k-step's other half is the neighbour's cell
    (1, 8, 8, (12, 40, 66), (3, 3, 3), 1),   # rows in parts
    (1, 16, 32, (9, 24, 64), (3, 3, 3), 2),  # epilogue teams that share a block
])
def test_infinities_and_nans_come_out_as_from_fp32_fma(geom, mode, value):
    """... and only where they are a term: the cells around keep their values (strides 2:
    an instruction also multiplies a cell with the zeros of taps that an output does not have)."""
    N, C, K, sp, f, s = geom
    if mode != _abi.MATH_FP32 and s == 1 and np.isinf(value):
        pytest.skip("one pass, stride 1: an infinity beside a zero may give a NaN")
    rng = np.random.default_rng(9)
    pads, strides, dil = [(e - 1) // 2 for e in f], [s] * len(sp), [1] * len(sp)
    x = rng.normal(size=(N, C, *sp)).astype(np.float32)
    w = rng.normal(size=(K, C, *f)).astype(np.float32)
    w[0] = 1.0  # exactly representable: no second part to meet an infinity
    dy = rng.normal(size=(N, K, *[O.conv_out_extent(i, e, (e - 1) // 2, s, 1) for i, e in zip(sp, f)])).astype(np.float32)
    for at in (tuple(e // 2 for e in sp), (0,) * len(sp), tuple(e - 1 for e in sp)):
        x[(0, C - 1) + at] = value
        dy[(0, K - 1) + tuple(min(a // s, e - 1) for a, e in zip(at, dy.shape[2:]))] = -value
    got = run_all(x, w, dy, pads, strides, dil, mode)
    with np.errstate(all="ignore"):
        ref = [O.conv_fwd(x, w, pads, strides), np.zeros_like(x), O.conv_bwd_filter(x, dy, f, pads, strides)]
        O.conv_bwd_data(w, dy, ref[1], pads, strides)
    for name, a, b in zip(("y", "dx", "dw"), got, ref):
        assert np.array_equal(np.isnan(a), np.isnan(b)), name
        assert np.array_equal(np.isposinf(a), np.isposinf(b)) and np.array_equal(np.isneginf(a), np.isneginf(b)), name
        assert np.isfinite(b).any()
        scale = np.sqrt(np.mean(np.square(b[np.isfinite(b)])))
        bound = 2e-5 if mode == _abi.MATH_FP32 or name == "dw" else 4e-2
        assert np.abs(a - b)[np.isfinite(b)].max() <= bound * (scale + np.abs(b[np.isfinite(b)]).max()), name


def test_statistics_of_an_output_with_an_infinity():
    """The statistics' epilogue sees the repaired values."""
    rng = np.random.default_rng(10)
    N, C, K, sp = 1, 4, 16, (6, 9, 33)
    x = torch.from_numpy(rng.normal(size=(N, C, *sp)).astype(np.float32)).cuda()
    w = torch.ones(K, C, 3, 3, 3, device="cuda")
    w[1:] = torch.from_numpy(rng.normal(size=(K - 1, C, 3, 3, 3)).astype(np.float32)).cuda()
    w[3, 1] = 0.0  # inf * 0
    x[0, 1, 3, 4, 5] = float("inf")
    y, sums = torch.empty(N, K, *sp, device="cuda"), torch.zeros(2, K, device="cuda")
    p = Plan(x, w, y, [1] * 3, [1] * 3, [1] * 3, _abi.MATH_FP32)
    assert _abi.lib().dcb_conv_fwd_stats(p.p, 1.0, x.data_ptr(), w.data_ptr(), y.data_ptr(), sums[0].data_ptr(),
                                         sums[1].data_ptr(), None) == _abi.OK
    torch.cuda.synchronize()
    assert torch.equal(torch.isnan(sums[0]), torch.isnan(y.sum((0, 2, 3, 4)))) and bool(torch.isnan(sums[0][3]))
    assert float(sums[0][0]) == float("inf") and float(sums[1][0]) == float("inf")


def _round_tf32(a):
    return ((a.view(np.uint32) + np.uint32(0x1000)) & np.uint32(0xFFFFE000)).view(np.float32)


@pytest.mark.parametrize("mode", [_abi.MATH_FP32, _abi.MATH_TF32, _abi.MATH_BF16])
@pytest.mark.parametrize("geom", [g for g, _ in layers.SWEEP])
def test_converters_of_the_sweep_kernel(geom, mode):
    """Every converter, alone and with statistics (to fp32 rounding of partial sums); one pass: the product of the rounded operands."""
    N, C, K, sp, f, pads = geom
    rng = np.random.default_rng(C + sp[-1])
    x = rng.normal(0.3, 1, (N, C, *sp)).astype(np.float32)
    w = rng.normal(0, np.sqrt(2.0 / (C * np.prod(f))), (K, C, *f)).astype(np.float32)
    xs, ws = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    y = torch.full((N, K, *[O.conv_out_extent(i, e, p, 1, 1) for i, e, p in zip(sp, f, pads)]), float("nan"), device="cuda")
    sums = torch.full((2, K), float("nan"), device="cuda")
    p = Plan(xs, ws, y, pads, [1] * 3, [1] * 3, mode)
    rnd = {_abi.MATH_FP32: lambda a: a, _abi.MATH_TF32: _round_tf32, _abi.MATH_BF16: _round_bf16}[mode]
    ref = O.conv_fwd(rnd(x), rnd(w), pads, [1] * 3)
    p.fwd(1.0, xs, ws, 0.0, y)
    emu.assert_close(y.cpu().numpy(), ref, TOL, "y")
    y.fill_(float("nan"))
    assert _abi.lib().dcb_conv_fwd_stats(p.p, 1.0, xs.data_ptr(), ws.data_ptr(), y.data_ptr(), sums[0].data_ptr(),
                                         sums[1].data_ptr(), None) == _abi.OK
    emu.assert_close(y.cpu().numpy(), ref, TOL, "y with statistics")
    assert _abi.lib().dcb_conv_plan_status(p.p, None) == _abi.OK
    d, over = y.double(), (0, 2, 3, 4)
    for got, exact, size in ((sums[0], d.sum(over), d.abs().sum(over)), (sums[1], d.square().sum(over), d.square().sum(over))):
        assert ((got.double() - exact).abs() <= 1e-5 * size).all()


@pytest.mark.parametrize("mode", [_abi.MATH_FP32, _abi.MATH_BF16])
@pytest.mark.parametrize("geom", [
    (1, 4, 16, (6, 9, 9), (3, 3, 3), 1),      # sub-columns side by side
    (2, 8, 7, (5, 11, 31), (3, 3, 3), 1),     # two samples, filters padded
    (1, 16, 16, (7, 9, 101), (3, 3, 3), 1),   # ragged rows: plain stores
    (1, 16, 4, (8, 9, 132), (3, 3, 3), 2),    # stride 2
    (1, 32, 16, (64, 64, 64), (3, 3, 3), 1),  # channel groups, in fp32 parts of rows
    layers.STATISTICS_BY_BULK_STORES,
])
def test_statistics_from_the_shift_kernel(geom, mode):
    """Sums and sums of squares of the output that it wrote, to fp32 rounding of partial sums:
    2^-24 per addition of a lane's chain, some hundred of them."""
    N, C, K, sp, f, s = geom
    gen = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(N, C, *sp, device="cuda", generator=gen) + 0.5
    w = torch.randn(K, C, *f, device="cuda", generator=gen) * 0.1
    y = torch.full((N, K, *[O.conv_out_extent(i, 3, 1, s, 1) for i in sp]), float("nan"), device="cuda")
    sums = torch.full((2, K), float("nan"), device="cuda")
    p = Plan(x, w, y, [1] * 3, [s] * 3, [1] * 3, mode)
    assert _abi.lib().dcb_conv_plan_kernel_kind(p.p, 0) == 1
    assert _abi.lib().dcb_conv_fwd_stats(p.p, 1.0, x.data_ptr(), w.data_ptr(), y.data_ptr(), sums[0].data_ptr(),
                                         sums[1].data_ptr(), None) == _abi.OK
    torch.cuda.synchronize()
    assert _abi.lib().dcb_conv_plan_status(p.p, None) == _abi.OK
    # not against dcb_conv_fwd's bits: the pipe truncates and the issuers' instructions land in an
    # order that varies from run to run, so that two plain forward passes differ in their last bits too
    xr, wr = (x, w) if mode == _abi.MATH_FP32 else (torch.from_numpy(_round_bf16(a.cpu().numpy())).cuda() for a in (x, w))
    ref = torch.nn.functional.conv3d(xr.double(), wr.double(), None, s, 1)
    emu.assert_close(y.cpu().numpy(), ref.cpu().numpy(), TOL, "y")
    d, over = y.double(), (0, 2, 3, 4)
    for got, ref, size in ((sums[0], d.sum(over), d.abs().sum(over)), (sums[1], d.square().sum(over), d.square().sum(over))):
        assert ((got.double() - ref).abs() <= 1e-5 * size).all()


@pytest.mark.parametrize("mode", [_abi.MATH_FP32, _abi.MATH_TF32, _abi.MATH_BF16])
@pytest.mark.parametrize("geom", [
    # N, C, K, spatial, filter, padding, stride: one tap along D, columns of several rows, several planes a CTA
    (3, 4, 3, (56, 51, 132), (1, 1, 1), (0, 0, 0), 1), (1, 8, 32, (40, 64, 64), (1, 2, 2), (0, 0, 0), 1),
    (1, 8, 8, (40, 64, 64), (1, 3, 3), (0, 1, 1), 2), (2, 16, 8, (60, 80, 64), (2, 2, 2), (0, 0, 0), 2),
])
def test_planes_that_open_and_close_in_one_step(geom, mode):
    N, C, K, sp, f, pads, s = geom
    rng = np.random.default_rng(K)
    rnd = {_abi.MATH_FP32: lambda a: a, _abi.MATH_TF32: _round_tf32, _abi.MATH_BF16: _round_bf16}[mode]
    x = rnd(rng.normal(size=(N, C, *sp)).astype(np.float32))
    w = rnd(rng.normal(0, np.sqrt(2.0 / (C * np.prod(f))), (K, C, *f)).astype(np.float32))
    dy = rnd(rng.normal(size=(N, K, *[O.conv_out_extent(i, e, p, s, 1) for i, e, p in zip(sp, f, pads)])).astype(np.float32))
    for _ in range(3):
        y, dx, dw = run_all(x, w, dy, pads, [s] * 3, [1] * 3, mode)
        emu.assert_close(y, O.conv_fwd(x, w, pads, [s] * 3), TOL, "y")
        dx_ref = np.zeros_like(x)
        O.conv_bwd_data(w, dy, dx_ref, pads, [s] * 3)
        emu.assert_close(dx, dx_ref, TOL, "dx")


@pytest.mark.parametrize("mode", [_abi.MATH_FP32, _abi.MATH_BF16])
@pytest.mark.parametrize("geom", [
    # N, C, K, spatial, filter, stride: rows that are laid side by side in parts, last parts short
    (1, 32, 24, (9, 33, 64), (3, 3, 3), 1), (2, 24, 28, (7, 20, 132), (3, 3, 3), 1), (1, 12, 20, (9, 31, 177), (3, 3, 3), 1),
    (1, 8, 8, (12, 40, 66), (3, 3, 3), 1), (2, 32, 16, (75, 65), (3, 3), 1), (1, 16, 24, (11, 23, 160), (3, 3, 3), 2),
] + layers.STRIDED_ROWS_IN_PARTS)
def test_rows_in_parts(geom, mode):
    N, C, K, sp, f, s = geom
    rng = np.random.default_rng(sp[-1])
    pads, strides = [1] * len(sp), [s] * len(sp)
    x = rng.normal(size=(N, C, *sp)).astype(np.float32)
    w = rng.normal(0, np.sqrt(2.0 / (C * np.prod(f))), (K, C, *f)).astype(np.float32)
    dy = rng.normal(size=(N, K, *[O.conv_out_extent(i, 3, 1, s, 1) for i in sp])).astype(np.float32)
    y, dx, _ = run_all(x, w, dy, pads, strides, [1] * len(sp), mode)
    if mode == _abi.MATH_BF16:  # exact products of rounded operands, fp32 sums
        x, w, dy = _round_bf16(x), _round_bf16(w), _round_bf16(dy)
    dx_ref = np.zeros_like(x)
    O.conv_bwd_data(w, dy, dx_ref, pads, strides)
    emu.assert_close(y, O.conv_fwd(x, w, pads, strides), TOL, "y")
    emu.assert_close(dx, dx_ref, TOL, "dx")


@pytest.mark.parametrize("beta", [0.0, 0.5])
@pytest.mark.parametrize("geom", [
    # N, C, K, spatial, filter, stride: columns of one row without a spare plane slot, blocks with two halves:
    # parities along W of 4 filters a cell, 16 + 12 and 16 + 16 filters (last part of a row short), W odd
    (1, 16, 32, (9, 24, 64), (3, 3, 3), 2), (1, 28, 32, (9, 20, 50), (3, 3, 3), 1), (2, 24, 28, (7, 20, 131), (3, 3, 3), 1),
    (1, 16, 32, (9, 24, 61), (3, 3, 3), 2),
])
def test_epilogue_teams_that_share_a_block(geom, beta):
    N, C, K, sp, f, s = geom
    rng = np.random.default_rng(sp[-1] + 1)
    pads, strides = [1] * len(sp), [s] * len(sp)
    out = [O.conv_out_extent(i, 3, 1, s, 1) for i in sp]
    x, dy, y0, dx0 = (rng.normal(size=(N, c, *e)).astype(np.float32) for c, e in ((C, sp), (K, out), (K, out), (C, sp)))
    w = rng.normal(0, np.sqrt(2.0 / (C * np.prod(f))), (K, C, *f)).astype(np.float32)
    y, dx, _ = run_all(x, w, dy, pads, strides, [1] * len(sp), _abi.MATH_FP32, 1.0, beta, y0.copy(), dx0.copy(), np.zeros_like(w))
    dx_ref = np.zeros_like(x)
    O.conv_bwd_data(w, dy, dx_ref, pads, strides)
    emu.assert_close(y, O.conv_fwd(x, w, pads, strides) + beta * y0, TOL, "y")
    emu.assert_close(dx, dx_ref + beta * dx0, TOL, "dx")


def test_epilogue_teams_that_share_a_block_of_16_filters_a_cell():
    """Large enough for all filters in one group; chains of 16 updates, 2^-25 of the result each, as much
    again for the rounding of the sums, 2^-22 for the split."""
    assert max(_relative_errors(1, 16, 32, (64, 128, 256), (3, 3, 3), 2, _abi.MATH_FP32)) <= 16 * 2.0 ** -25 + 2.0 ** -22


@pytest.mark.parametrize("geom", [
    # N, C, K, spatial, filter, stride: operands whose rows do not fill a multiple of 8, or a tile's 128
    (1, 3, 13, (9, 11, 37), (3, 3, 3), 1), (2, 5, 3, (30, 41), (5, 5), 1), (1, 4, 16, (16, 24, 32), (3, 3, 3), 1), (1, 7, 9, (8, 9, 34), (3, 3, 3), 2),
])
def test_backward_filter_behind_one_of_nans(geom):
    """What an earlier kernel left in shared and tensor memory reaches no output."""
    N, C, K, sp, f, s = geom
    rng = np.random.default_rng(K)
    pads, strides = [(e - 1) // 2 for e in f], [s] * len(sp)
    x = rng.normal(size=(N, C, *sp)).astype(np.float32)
    dy = rng.normal(size=(N, K, *[O.conv_out_extent(i, e, p, s, 1) for i, e, p in zip(sp, f, pads)])).astype(np.float32)
    xs, dys, dw = torch.from_numpy(x).cuda(), torch.from_numpy(dy).cuda(), torch.zeros(K, C, *f, device="cuda")
    p = Plan(xs, dw, dys, pads, strides, [1] * len(sp), _abi.MATH_FP32)
    assert _abi.lib().dcb_conv_plan_kernel_kind(p.p, 2) == 1
    p.bwd_filter(1.0, torch.full_like(xs, float("nan")), torch.full_like(dys, float("nan")), 0.0, dw)
    assert bool(torch.isnan(dw).all())
    p.bwd_filter(1.0, xs, dys, 0.0, dw)
    emu.assert_close(dw.cpu().numpy(), O.conv_bwd_filter(x, dy, f, pads, strides), TOL, "dw")
