"""Pooling kernels against the oracle, through the C ABI and through the
Pooling operator on emulated ranks (halo exchange forward, reverse exchange
with SUM backward)."""
import ctypes

import numpy as np
import pytest
import torch

import dihydrogen_b200 as dc
from dihydrogen_b200 import _abi
from oracle import oracle as O

import emu
from test_gpu_conv import _nd

pytestmark = pytest.mark.gpu

MODES = list(_abi.POOL_MODES)

# N, C, spatial extents, window, pads, strides
CASES = [
    (2, 3, (7, 9, 11), (3, 3, 3), (1, 1, 1), (2, 2, 2)),
    (1, 2, (8, 10), (2, 2), (0, 0), (2, 2)),
    (2, 2, (6, 7, 8), (3, 3, 3), (1, 1, 1), (1, 1, 1)),
    (1, 2, (9, 300), (3, 3), (0, 0), (1, 1)),
    (1, 1, (4, 6, 520), (2, 2, 2), (0, 0, 0), (2, 2, 2)),
    (1, 2, (11, 13), (5, 5), (2, 2), (3, 3)),
    # long rows of window 3 / stride 2 / pad 1: the four-cells-per-thread backward pass over several warps
    (1, 2, (5, 6, 260), (3, 3, 3), (1, 1, 1), (2, 2, 2)),
    (1, 2, (9, 64), (3, 3), (1, 1), (2, 2)),
    (1, 1, (4, 5, 131), (3, 3, 3), (0, 1, 1), (2, 2, 2)),
    # even extents everywhere: every thread of the 2 x 2-rows backward pass owns a whole block
    (1, 2, (6, 8, 72), (3, 3, 3), (1, 1, 1), (2, 2, 2)),
]


def _pd(window, pads, strides, mode):
    nsd = len(window)
    pd = _abi.PoolDesc()
    pd.nsd, pd.mode = nsd, _abi.POOL_MODES[mode]
    for i in range(3):
        pd.window[i], pd.pads[i], pd.strides[i] = 1, 0, 1
    for i in range(nsd):
        pd.window[3 - nsd + i], pd.pads[3 - nsd + i], pd.strides[3 - nsd + i] = window[i], pads[i], strides[i]
    return pd


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("case", CASES)
def test_kernels_against_oracle(case, mode):
    N, C, sp, window, pads, strides = case
    rng = np.random.default_rng(3)
    # small integers: ties inside windows, so that "first maximum" matters
    x = rng.integers(-4, 5, size=(N, C, *sp)).astype(np.float32)
    y_ref = O.pool_fwd(x, window, pads, strides, mode)
    dy = rng.normal(size=y_ref.shape).astype(np.float32)
    dx_ref = O.pool_bwd(x, dy, window, pads, strides, mode)
    xs, dys = torch.from_numpy(x).cuda(), torch.from_numpy(dy).cuda()
    y0 = rng.normal(size=y_ref.shape).astype(np.float32)
    dx0 = rng.normal(size=x.shape).astype(np.float32)
    y, dx = torch.zeros_like(dys), torch.zeros_like(xs)
    pd, xd, yd = _pd(window, pads, strides, mode), _nd(xs), _nd(y)
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    _abi.call("dcb_pool_fwd", ctypes.byref(pd), ctypes.byref(xd), ctypes.byref(yd), 1.0, P(xs), 0.0, P(y), None)
    _abi.call("dcb_pool_bwd", ctypes.byref(pd), ctypes.byref(xd), ctypes.byref(yd), 1.0, P(y), P(dys), P(xs), 0.0,
              P(dx), None, 0, None)
    torch.cuda.synchronize()
    emu.assert_close(y.cpu().numpy(), y_ref, 1e-6, "y")
    emu.assert_close(dx.cpu().numpy(), dx_ref, 2e-6, "dx")
    # with the index workspace: the same gradient, bit for bit
    need = _abi.lib().dcb_pool_bwd_workspace_bytes(ctypes.byref(pd), ctypes.byref(xd), ctypes.byref(yd))
    assert need == (y.numel() if mode == "MAX" else 0)
    if need:
        ws = torch.empty(need, dtype=torch.uint8, device="cuda")
        dx2 = torch.full_like(xs, 9.0)
        _abi.call("dcb_pool_bwd", ctypes.byref(pd), ctypes.byref(xd), ctypes.byref(yd), 1.0, P(y), P(dys), P(xs), 0.0,
                  P(dx2), P(ws), need, None)
        torch.cuda.synchronize()
        assert torch.equal(dx2, dx)
    # alpha / beta
    yb, dxb = torch.from_numpy(y0).cuda(), torch.from_numpy(dx0).cuda()
    _abi.call("dcb_pool_fwd", ctypes.byref(pd), ctypes.byref(xd), ctypes.byref(yd), 0.5, P(xs), 2.0, P(yb), None)
    _abi.call("dcb_pool_bwd", ctypes.byref(pd), ctypes.byref(xd), ctypes.byref(yd), 0.5, P(y), P(dys), P(xs), -1.0,
              P(dxb), None, 0, None)
    torch.cuda.synchronize()
    emu.assert_close(yb.cpu().numpy(), 0.5 * y_ref + 2.0 * y0, 2e-6, "y blend")
    emu.assert_close(dxb.cpu().numpy(), 0.5 * dx_ref - dx0, 4e-6, "dx blend")


# rows around multiples of four and of a block's shares of rows, padding on either side, gaps
# between windows, a window of each compiled kind and a general one; tensors as small as these
# take one output and one cell a thread (the larger ones follow)
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("window,pad,stride,widths", [
    (2, 0, 2, (2, 3, 8, 9, 10, 17, 66)),
    (3, 1, 1, (1, 2, 4, 5, 7, 16, 33, 1025)),
    (3, 1, 2, (1, 5, 6, 7, 9, 33, 35)),
    (2, 0, 3, (5, 8, 13)),
    (4, 2, 2, (3, 8, 21)),
])
def test_rows_of_all_lengths(window, pad, stride, widths, mode):
    for w in widths:
        for sp in ((5, 4, w), (6, w)):
            if min(sp) + 2 * pad >= window:
                test_kernels_against_oracle((1, 2, sp, *([v] * len(sp) for v in (window, pad, stride))), mode)


# the same rows where there are more than 32768 cells: backward, four cells a thread, and from 129 on a row a block
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("window,pad,stride,widths", [
    (2, 0, 2, (3, 8, 9, 129, 258)), (3, 1, 1, (4, 5, 17, 130)), (3, 1, 2, (5, 7, 18, 131, 257)), (4, 2, 2, (3, 8, 133)),
])
def test_rows_of_all_lengths_in_larger_tensors(window, pad, stride, widths, mode):
    for w in widths:
        sp = (33, -(-32769 // (2 * 33 * w)) + window, w)
        test_kernels_against_oracle((1, 2, sp, *([v] * 3 for v in (window, pad, stride))), mode)
    test_kernels_against_oracle((1, 2, (-(-32769 // (2 * widths[-1])) + window, widths[-1]), *([v] * 2 for v in (window, pad, stride))), mode)


# outputs a thread: two and four (fewer than 65537 outputs, as everywhere else here, take one)
MANY_OUTPUTS = [
    (1, 4, (42, 43, 81), (2, 2, 2), (0, 0, 0), (2, 2, 2)),    # two, stride 2: 70560 outputs
    (1, 7, (21, 71, 89), (3, 3, 3), (1, 1, 1), (2, 2, 2)),    # two, rows off 16-byte boundaries
    (2, 5, (131, 257), (3, 3), (0, 0), (2, 2)),               # two, images
    (2, 16, (30, 50, 53), (2, 2, 2), (0, 0, 0), (2, 2, 2)),   # four, stride 2: 312000 outputs in short rows
    (1, 3, (16, 31, 46), (3, 3, 3), (1, 1, 1), (1, 1, 1)),    # four, stride 1: 68448 outputs
    (3, 2, (111, 101), (3, 3), (1, 1), (1, 1)),
]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("case", MANY_OUTPUTS)
def test_many_outputs(case, mode):
    test_kernels_against_oracle(case, mode)


@pytest.mark.parametrize("case", MANY_OUTPUTS + [
    (2, 2, (5, 6, 7), (2, 2, 2), (0, 0, 0), (2, 2, 2)), (1, 2, (5, 8, 9), (3, 3, 3), (1, 1, 1), (2, 2, 2)),
    (1, 2, (4, 9, 33), (3, 3, 3), (1, 1, 1), (1, 1, 1)), (2, 2, (13, 6), (3, 3), (1, 1), (1, 1)),
])
def test_maxima_of_infinities_and_nans(case):
    """A window's cells in order: the first one, whatever it is, then every one that is greater."""
    N, C, sp, window, pads, strides = case
    rng = np.random.default_rng(5)
    x = rng.integers(-3, 3, size=(N, C, *sp)).astype(np.float32)
    u = rng.random(x.shape)
    for lo, value in ((.1, -np.inf), (.3, np.float32(-3.4028234663852886e38)), (.5, np.nan), (.6, np.inf), (.7, -0.0)):
        x[(u > lo) & (u < lo + .08)] = value
    x[:, 0, :3] = -np.inf
    nsd = len(sp)
    w3, p3, s3 = ([a] * (3 - nsd) + list(v) for a, v in ((1, window), (0, pads), (1, strides)))
    vals, where, out = O._pool_windows(O._as5(x), w3, p3, s3)
    r, best = np.full(vals.shape[1:], -3.4028234663852886e38), np.full(vals.shape[1:], -1)
    for v, at in zip(vals, where):
        with np.errstate(invalid="ignore"):
            take = (at >= 0) & ((best < 0) | (v > r))
        r, best = np.where(take, v, r), np.where(take, at, best)
    xs = torch.from_numpy(x).cuda()
    y = torch.zeros((N, C, *out[3 - nsd:]), device="cuda")
    dys, dx = torch.randn_like(y), torch.full_like(xs, 9.0)
    pd, xd, yd = _pd(window, pads, strides, "MAX"), _nd(xs), _nd(y)
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    _abi.call("dcb_pool_fwd", ctypes.byref(pd), ctypes.byref(xd), ctypes.byref(yd), 1.0, P(xs), 0.0, P(y), None)
    ws = torch.empty(y.numel(), dtype=torch.uint8, device="cuda")
    _abi.call("dcb_pool_bwd", ctypes.byref(pd), ctypes.byref(xd), ctypes.byref(yd), 1.0, P(y), P(dys), P(xs), 0.0, P(dx),
              P(ws), ws.numel(), None)
    assert np.array_equal(y.cpu().numpy().reshape(r.shape), r.astype(np.float32), equal_nan=True)
    dx_ref = np.zeros((N, C, x[0, 0].size))
    for i in range(N):
        for j in range(C):
            np.add.at(dx_ref[i, j], best[i, j].ravel(), dys[i, j].cpu().numpy().ravel())
    emu.assert_close(dx.cpu().numpy(), dx_ref.reshape(x.shape).astype(np.float32), 2e-6, "dx")


# window 3, stride 2: walks of several outputs along D (the last one shorter), one walk
# per output, an odd row end, no padding along D
@pytest.mark.parametrize("n,c,sp,pad_d", [(1, 512, (37, 31, 20), 1), (2, 512, (24, 9, 8), 0), (1, 2, (6, 5, 264), 1),
                                          (1, 3, (1, 2, 8), 1)])
def test_walk_along_depth(n, c, sp, pad_d):
    rng = np.random.default_rng(9)
    window, pads, strides = (3, 3, 3), (pad_d, 1, 1), (2, 2, 2)
    x = rng.integers(-4, 5, size=(n, c, *sp)).astype(np.float32)
    x[rng.random(x.shape) < 0.2] = np.nan  # a window's first cell that is no number stays its maximum
    x[rng.random(x.shape) < 0.1] = -np.inf
    o = [(e + 2 * p - 3) // 2 + 1 for e, p in zip(sp, pads)]
    # the rule in words: cells in D, H, W order, the first becomes the maximum, a later one if it is larger
    best, idx = np.full((n, c, *o), np.nan, np.float32), np.full((n, c, *o), -1)
    total = np.zeros((n, c, *o))
    at = np.meshgrid(*[np.arange(e) * 2 for e in o], indexing="ij")
    for kd in range(3):
        for kh in range(3):
            for kw in range(3):
                q = [a + k - p for a, k, p in zip(at, (kd, kh, kw), pads)]
                ok = np.logical_and.reduce([(a >= 0) & (a < e) for a, e in zip(q, sp)])
                v = x[:, :, *[np.clip(a, 0, e - 1) for a, e in zip(q, sp)]]
                with np.errstate(invalid="ignore"):
                    take = ok & ((idx < 0) | (v > best))
                best, idx = np.where(take, v, best), np.where(take, np.ravel_multi_index(
                    [np.clip(a, 0, e - 1) for a, e in zip(q, sp)], sp), idx)
                total += np.where(ok & np.isfinite(v), v, 0)
    dy = rng.integers(-8, 9, size=best.shape).astype(np.float32)  # whole numbers: sums are exact in any order
    dx_ref = np.zeros((n * c, int(np.prod(sp))), np.float32)
    np.add.at(dx_ref, (np.arange(n * c)[:, None], idx.reshape(n * c, -1)), dy.reshape(n * c, -1))
    xs, dys = torch.from_numpy(x).cuda(), torch.from_numpy(dy).cuda()
    y, dx = torch.zeros_like(dys), torch.zeros_like(xs)
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    pd, xd, yd = _pd(window, pads, strides, "MAX"), _nd(xs), _nd(y)
    _abi.call("dcb_pool_fwd", ctypes.byref(pd), ctypes.byref(xd), ctypes.byref(yd), 1.0, P(xs), 0.0, P(y), None)
    ws = torch.empty(y.numel(), dtype=torch.uint8, device="cuda")
    _abi.call("dcb_pool_bwd", ctypes.byref(pd), ctypes.byref(xd), ctypes.byref(yd), 1.0, P(y), P(dys), P(xs), 0.0,
              P(dx), P(ws), ws.numel(), None)
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy(), best, equal_nan=True)
    assert np.array_equal(dx.cpu().numpy().reshape(dx_ref.shape), dx_ref)
    # averages: whole numbers, so the sums are exact and one division rounds
    pd, xf = _pd(window, pads, strides, "AVERAGE"), torch.from_numpy(np.where(np.isfinite(x), x, 0)).cuda()
    _abi.call("dcb_pool_fwd", ctypes.byref(pd), ctypes.byref(xd), ctypes.byref(yd), 1.0, P(xf), 0.0, P(y), None)
    torch.cuda.synchronize()
    assert np.allclose(y.cpu().numpy(), total / 27, rtol=2.0 ** -23, atol=0)


def test_rejects_mismatched_output_extent():
    x = torch.zeros(1, 1, 8, 8, device="cuda")
    y = torch.zeros(1, 1, 5, 4, device="cuda")
    pd, xd, yd = _pd((2, 2), (0, 0), (2, 2), "MAX"), _nd(x), _nd(y)
    st = _abi.lib().dcb_pool_fwd(ctypes.byref(pd), ctypes.byref(xd), ctypes.byref(yd), 1.0,
                                 ctypes.c_void_p(x.data_ptr()), 0.0, ctypes.c_void_p(y.data_ptr()), None)
    assert st == _abi.BAD_ARG


# global shape (W, H, [D,] C, N), locale, window, pad, stride
PARTITIONED = [
    ([20, 16, 12, 3, 2], [1, 1, 4, 1, 1], 3, 1, 1),
    ([16, 16, 16, 2, 1], [2, 2, 2, 1, 1], 3, 1, 2),
    ([24, 20, 3, 2], [2, 2, 1, 1], 3, 1, 1),
    ([16, 12, 8, 2, 1], [1, 2, 2, 1, 1], 2, 0, 2),
    ([18, 14, 10, 2, 1], [1, 2, 2, 1, 1], 3, 0, 1),
]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("shape,locale,window,pad,stride", PARTITIONED)
def test_partitioned_pooling_matches_single_domain(shape, locale, window, pad, stride, mode):
    nd = len(shape)
    nsd = nd - 2
    n = int(np.prod(locale))
    bes = emu.make_backends(n)
    win, pads, strides = [window] * nsd, [pad] * nsd, [stride] * nsd
    rng = np.random.default_rng(5)
    gx = rng.integers(-4, 5, size=tuple(reversed(shape))).astype(np.float32)
    y_ref = O.pool_fwd(gx, win, pads, strides, mode)
    gdy = rng.normal(size=y_ref.shape).astype(np.float32)
    dx_ref = O.pool_bwd(gx, gdy, win, pads, strides, mode)
    xs, ys, dxs, dys, pools = [], [], [], [], []
    for be in bes:
        x = dc.create_input_tensor(shape, locale, win, strides, [1] * nsd, be.locale)
        y = dc.create_pooling_output_tensor(x, win, strides, pads)
        dx = dc.create_d_input_tensor(x)
        dy = dc.create_pooling_d_output_tensor(y)
        for t in (x, y, dx, dy):
            t.allocate()
        emu.scatter_owned(x, gx)
        own = x.owned().clone()
        x.buffer.fill_(float("nan"))  # halos must be produced by the exchange
        x.owned().copy_(own)
        dx.buffer.fill_(float("nan"))  # and every cell of dx by the backward pass
        emu.scatter_owned(dy, gdy)
        pool = dc.Pooling(be, nd)
        pool.setup(x, y, dx, dy, win, pads, strides, mode, connect=False)
        xs.append(x), ys.append(y), dxs.append(dx), dys.append(dy), pools.append(pool)
    assert list(ys[0].shape) == list(reversed(y_ref.shape))
    emu.connect_halo([p.halo_xch_input for p in pools])
    emu.connect_halo([p.halo_xch_d_input for p in pools])
    for x in xs:
        for d in range(nsd):
            x.clear_halo(d)
    emu.exchange_all([p.halo_xch_input for p in pools])
    for p, x, y in zip(pools, xs, ys):
        p.forward(1.0, x, 0.0, y, skip_halo_exchange=True)
    for p, x, y, dx, dy in zip(pools, xs, ys, dxs, dys):
        p.backward(1.0, y, dy, x, 0.0, dx, skip_halo_exchange=True)
    emu.exchange_all([p.halo_xch_d_input for p in pools], is_reverse=True, op="SUM")
    torch.cuda.synchronize()
    emu.assert_close(emu.gather_owned(ys, y_ref.shape), y_ref, 1e-6, "y")
    emu.assert_close(emu.gather_owned(dxs, gx.shape), dx_ref, 4e-6, "dx")
