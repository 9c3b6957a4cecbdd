"""Batch-norm kernels against the oracle (fp32, 1e-5 relative)."""
import numpy as np
import pytest
import torch

import dihydrogen_b200 as dc
from dihydrogen_b200 import _abi
from oracle import oracle as O

import emu

pytestmark = pytest.mark.gpu

TOL = 1e-5

# shape (W..N), locale, overlap: dense, D-halo (contiguous planes), H/W halos
# (strided rows), odd extents (scalar path)
CASES = [
    ([32, 16, 8, 4, 2], [1, 1, 1, 1, 1], [0, 0, 0, 0, 0]),
    ([32, 16, 8, 4, 2], [1, 1, 2, 1, 1], [0, 0, 1, 0, 0]),
    ([32, 16, 8, 4, 1], [2, 2, 2, 1, 1], [1, 1, 1, 0, 0]),
    ([33, 7, 5, 3, 2], [1, 1, 1, 1, 1], [0, 0, 0, 0, 0]),
    ([34, 9, 6, 2], [1, 2, 1, 1], [0, 2, 0, 0]),
    ([130, 129, 3, 1], [1, 1, 1, 1], [0, 0, 0, 0]),
    ([64, 64, 64, 16, 1], [1, 1, 1, 1, 1], [0, 0, 0, 0, 0]),
    # W halo: padded rows, a unit of the kernels packs several rows (16 + 16 + 5 of a plane's 37)
    ([512, 37, 3, 4, 1], [2, 1, 1, 1, 1], [1, 0, 0, 0, 0]),
    ([32, 50, 3, 2, 1], [2, 1, 1, 1, 1], [1, 0, 0, 0, 0]),
]


def _rank0(shape, locale, overlap):
    n = int(np.prod(locale))
    return dc.Tensor(shape, dc.Locale(0, n), dc.Distribution.make_overlapped_distribution(locale, overlap))


@pytest.mark.parametrize("shape,locale,overlap", CASES)
def test_bn_forward_backward_local(shape, locale, overlap):
    rng = np.random.default_rng(3)
    be = dc.BackendDNNLib(dc.Locale(0, 1))
    x_t, y_t, dy_t, dx_t = (_rank0(shape, locale, overlap) for _ in range(4))
    real = x_t.np_real_shape()
    C = shape[-2]
    xb = rng.normal(0.3, 1.5, real).astype(np.float32)
    dyb = rng.normal(0, 1, real).astype(np.float32)
    emu.upload(x_t, xb)
    emu.upload(dy_t, dyb)
    y_t.allocate()
    dx_t.allocate()
    own = O.Shard(shape, locale, overlap, 0).owned_slices()
    x, dy = xb[own], dyb[own]

    bn = dc.BatchNormalization(be, len(shape), decay=0.9, epsilon=1e-5, global_stats=False)
    stats = torch.zeros(2 * C, device="cuda")
    mean, var = stats[:C], stats[C:]
    rm, rv = torch.zeros(C, device="cuda"), torch.ones(C, device="cuda")
    scale = torch.from_numpy(rng.uniform(0.5, 1.5, C).astype(np.float32)).cuda()
    bias = torch.from_numpy(rng.normal(0, 1, C).astype(np.float32)).cuda()

    bn.forward_stage1(x_t, mean, var, True)
    s, q = O.bn_sums(x)
    emu.assert_close(mean.cpu().numpy(), s, TOL, "sums")
    emu.assert_close(var.cpu().numpy(), q, TOL, "sqsums")
    bn.forward_stage2(x_t, mean, var, rm, rv, scale, bias, y_t, True)
    nps = x.size // C
    m_ref, v_ref, rm_ref, rv_ref = O.bn_sums_to_statistics(s, q, nps, 0.9, np.zeros(C), np.ones(C))
    emu.assert_close(mean.cpu().numpy(), m_ref, TOL, "mean")
    emu.assert_close(var.cpu().numpy(), v_ref, 2e-5, "var")
    emu.assert_close(rm.cpu().numpy(), rm_ref, TOL, "running_mean")
    emu.assert_close(rv.cpu().numpy(), rv_ref, TOL, "running_var")
    # apply is checked with the GPU's own statistics so only its arithmetic is compared
    m_g, v_g = mean.cpu().numpy(), var.cpu().numpy()
    y_ref = O.bn_normalize(x, m_g, v_g, scale.cpu().numpy(), bias.cpu().numpy(), 1e-5)
    emu.assert_close(y_t.owned().cpu().numpy(), y_ref, TOL, "y")
    # halo cells of the output are untouched
    mask = np.ones(real, bool)
    mask[own] = False
    assert not y_t.buffer.cpu().numpy()[mask].any()

    grads = [torch.zeros(C, device="cuda") for _ in range(4)]
    dscale, dbias, dmean, dvar = grads
    bn.backward_stage1(x_t, dy_t, mean, var, scale, dscale, dbias, dmean, dvar)
    ref = O.bn_backprop1(x, dy, m_g, v_g, scale.cpu().numpy(), 1e-5)
    for g, r, nme in zip(grads, ref, ("dscale", "dbias", "dmean", "dvar")):
        emu.assert_close(g.cpu().numpy(), r, 2e-5, nme)
    bn.backward_stage2(x_t, dy_t, mean, var, scale, dmean, dvar, dx_t)
    dx_ref = O.bn_backprop2(x, dy, m_g, v_g, scale.cpu().numpy(), dmean.cpu().numpy(), dvar.cpu().numpy(), 1e-5, nps)
    emu.assert_close(dx_t.owned().cpu().numpy(), dx_ref, TOL, "dx")


@pytest.mark.parametrize("shape", [
    [41, 25, 1, 3, 2],   # 1025 elements a plane: just long enough for the statistics in pieces of four, every start
    [89, 23, 1, 3, 2],   # 2047 and 2049: on either side of what is long enough for the backward sums
    [683, 3, 1, 3, 2],
    [321, 17, 1, 3, 1],  # 5457 and 5459: on either side of eight pieces a thread
    [103, 53, 1, 4, 1],
    [91, 89, 1, 5, 1],   # 8099: the pieces of one or two units and the last, partial one
    [91, 91, 1, 4, 2],   # 8281: a last unit of 23 pieces
    [67, 83, 3, 2, 2],
])
def test_planes_of_odd_size(shape):
    test_bn_forward_backward_local(shape, [1] * 5, [0] * 5)


def test_several_long_runs_a_plane_that_start_anywhere():
    """A halo in H of odd rows: a run of 5561 elements per (n, c, d), each with a start of its own."""
    test_bn_forward_backward_local([67, 166, 3, 2, 2], [1, 2, 1, 1, 1], [0, 1, 0, 0, 0])


@pytest.mark.parametrize("x_off,dy_off", [(0, 0), (1, 1), (3, 3), (0, 2), (1, 2), (3, 0)])
def test_sums_of_planes_of_odd_size_wherever_they_lie(x_off, dy_off):
    """Both tensors alike: in pieces of four; not alike: element by element."""
    shape = [67, 83, 3, 3, 2]
    rng = np.random.default_rng(10 * x_off + dy_off)
    be, C = dc.BackendDNNLib(dc.Locale(0, 1)), shape[-2]
    x_t, dy_t = (_rank0(shape, [1] * 5, [0] * 5) for _ in range(2))
    emu.allocate_off_boundary(x_t, x_off)
    emu.allocate_off_boundary(dy_t, dy_off)
    x = rng.normal(0.3, 1.5, x_t.np_real_shape()).astype(np.float32)
    dy = rng.normal(0.1, 1, x.shape).astype(np.float32)
    x_t.buffer.copy_(torch.from_numpy(x))
    dy_t.buffer.copy_(torch.from_numpy(dy))
    bn = dc.BatchNormalization(be, 5, decay=0.9, epsilon=1e-5, global_stats=False)
    st, g = torch.zeros(2 * C, device="cuda"), torch.zeros(4 * C, device="cuda")
    bn.forward_stage1(x_t, st[:C], st[C:], True)
    for got, ref, name in zip(st.split(C), O.bn_sums(x), ("sums", "sqsums")):
        emu.assert_close(got.cpu().numpy(), ref, TOL, name)
    mean, var = x.mean(axis=(0, 2, 3, 4)), x.var(axis=(0, 2, 3, 4))
    scale = rng.uniform(0.5, 1.5, C).astype(np.float32)
    bn.backward_stage1(x_t, dy_t, *(torch.from_numpy(v).cuda() for v in (mean, var, scale)), *g.split(C))
    for got, ref, name in zip(g.split(C), O.bn_backprop1(x, dy, mean, var, scale, 1e-5), ("dscale", "dbias", "dmean", "dvar")):
        emu.assert_close(got.cpu().numpy(), ref, 2e-5, name)


def test_ends_of_unaligned_runs_are_summed_with_their_half():
    """A plane of 1800 pieces of four and three elements, in one unit of the statistics: the thread that has
    those three in the second half of its eight pieces has large values that cancel in the first."""
    H, W = 49, 147  # 7203
    be = dc.BackendDNNLib(dc.Locale(0, 1))
    x_t, dy_t = (_rank0([W, H, 1, 1], [1] * 4, [0] * 4) for _ in range(2))
    big = np.zeros(H * W, np.float32)
    big[:4096:2], big[1:4096:2] = 2.0 ** 26, -(2.0 ** 26)
    big[7200:] = 1.0
    for t in (x_t, dy_t):
        emu.upload(t, big.reshape(1, 1, H, W))
    bn = dc.BatchNormalization(be, 4, decay=0.9, epsilon=1e-5, global_stats=False)
    sums = torch.zeros(2, device="cuda")
    bn.forward_stage1(x_t, sums[:1], sums[1:], True)
    mean, var, scale = torch.zeros(1, device="cuda"), torch.ones(1, device="cuda"), torch.ones(1, device="cuda")
    grads = [torch.zeros(1, device="cuda") for _ in range(4)]
    bn.backward_stage1(x_t, dy_t, mean, var, scale, *grads)
    assert sums[0].item() == 3.0 and grads[1].item() == 3.0  # exact: powers of two and small whole numbers


@pytest.mark.parametrize("shape,overlap", [
    ([1, 1, 2, 1], [0, 0, 0, 0]),                  # one block per channel, two values
    ([33, 7, 5, 3, 2], [0, 0, 0, 0, 0]),
    ([128, 64, 64, 5, 1], [0, 0, 0, 0, 0]),        # several blocks per channel
    ([512, 37, 3, 4, 1], [0, 0, 0, 0, 0]),
])
@pytest.mark.parametrize("slope", [None, 0.25])
def test_finalize_inside_apply_equals_finalize_then_apply(shape, overlap, slope):
    """One launch or two: the same operations in the same order, so bit for bit the same."""
    rng = np.random.default_rng(11)
    be = dc.BackendDNNLib(dc.Locale(0, 1))
    x_t, y_t = (_rank0(shape, [1] * len(shape), overlap) for _ in range(2))
    emu.upload(x_t, rng.normal(0.3, 1.5, x_t.np_real_shape()).astype(np.float32))
    y_t.allocate()
    C = shape[-2]
    nps = int(np.prod(shape)) // C
    scale = torch.from_numpy(rng.uniform(0.5, 1.5, C).astype(np.float32)).cuda()
    bias = torch.from_numpy(rng.normal(0, 1, C).astype(np.float32)).cuda()
    bn = dc.BatchNormalization(be, len(shape), decay=0.9, epsilon=1e-5, global_stats=False)
    runs = []
    for fused in (False, True, True):  # twice: the tickets are back at zero
        mean, var, rm = (torch.zeros(C, device="cuda") for _ in range(3))
        rv = torch.ones(C, device="cuda")
        bn.forward_stage1(x_t, mean, var, True)
        if fused:
            bn.forward_stage2(x_t, mean, var, rm, rv, scale, bias, y_t, True, leaky_relu_slope=slope)
        else:
            _abi.call("dcb_bn_finalize", C, nps, 0.9, mean.data_ptr(), var.data_ptr(), rm.data_ptr(), rv.data_ptr(),
                      torch.cuda.current_stream().cuda_stream)
            # statistics given: apply only, as in inference
            bn.forward_stage2(x_t, mean, var, mean, var, scale, bias, y_t, False, leaky_relu_slope=slope)
        torch.cuda.synchronize()
        runs.append([t.cpu().numpy().tobytes() for t in (mean, var, rm, rv)] + [y_t.owned().cpu().numpy().tobytes()])
    assert runs[1] == runs[0] and runs[2] == runs[0]


def test_bn_stats_are_reproducible():
    """Fixed-order two-stage reduction: identical bits run to run."""
    shape = [64, 64, 32, 8, 1]
    t = _rank0(shape, [1] * 5, [0] * 5)
    emu.upload(t, np.random.default_rng(0).normal(size=t.np_real_shape()).astype(np.float32))
    be = dc.BackendDNNLib(dc.Locale(0, 1))
    bn = dc.BatchNormalization(be, 5, 0.9, 1e-5, False)
    outs = []
    for _ in range(3):
        st = torch.zeros(16, device="cuda")
        bn.forward_stage1(t, st[:8], st[8:], True)
        outs.append(st.cpu().numpy().copy())
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])


@pytest.mark.parametrize("locale", [[1, 1, 2, 1, 1], [2, 2, 2, 1, 1]])
def test_bn_global_stats_emulated_ranks(locale):
    """Distributed BN == single-rank BN (the reference's own criterion,
    legacy/tests/dnn_backend/test_cudnn_util.sh.in:387-425): per-channel sums
    all-reduced across the spatial partition."""
    shape = [16, 12, 10, 4, 2]
    C = 4
    rng = np.random.default_rng(5)
    g = rng.normal(0.1, 2.0, tuple(reversed(shape))).astype(np.float32)
    gdy = rng.normal(0, 1, g.shape).astype(np.float32)
    n = int(np.prod(locale))
    bes = emu.make_backends(n)
    dist = dc.Distribution.make_distribution(locale)
    xs, ys, dys, dxs = ([dc.Tensor(shape, b.locale, dist) for b in bes] for _ in range(4))
    for x, dy, y, dx in zip(xs, dys, ys, dxs):
        emu.scatter_owned(x, g)
        emu.scatter_owned(dy, gdy)
        y.allocate()
        dx.allocate()
    bns = [dc.BatchNormalization(b, 5, 0.9, 1e-5, True) for b in bes]
    stats = [torch.zeros(2 * C, device="cuda") for _ in bes]
    rms = [torch.zeros(C, device="cuda") for _ in bes]
    rvs = [torch.ones(C, device="cuda") for _ in bes]
    scale = torch.from_numpy(rng.uniform(0.5, 1.5, C).astype(np.float32)).cuda()
    bias = torch.from_numpy(rng.normal(0, 1, C).astype(np.float32)).cuda()
    for bn, x, st in zip(bns, xs, stats):
        bn.forward_stage1(x, st[:C], st[C:], True)
    emu.allreduce_all(bes, stats)
    for bn, x, y, st, rm, rv in zip(bns, xs, ys, stats, rms, rvs):
        bn.forward_stage2(x, st[:C], st[C:], rm, rv, scale, bias, y, True)
    s, q = O.bn_sums(g)
    nps = g.size // C
    m_ref, v_ref, _, _ = O.bn_sums_to_statistics(s, q, nps, 0.9, np.zeros(C), np.ones(C))
    y_ref = O.bn_normalize(g, m_ref, v_ref, scale.cpu().numpy(), bias.cpu().numpy(), 1e-5)
    for st in stats:  # every rank holds identical statistics
        assert np.array_equal(st.cpu().numpy(), stats[0].cpu().numpy())
    emu.assert_close(stats[0][:C].cpu().numpy(), m_ref, 1e-5, "mean")
    emu.assert_close(stats[0][C:].cpu().numpy(), v_ref, 2e-5, "var")
    emu.assert_close(emu.gather_owned(ys, g.shape), y_ref, 2e-5, "y")
    # backward
    g4 = [[torch.zeros(2 * C, device="cuda") for _ in bes] for _ in range(2)]  # (dmean|dvar), (dscale|dbias)
    for bn, x, dy, st, a, b in zip(bns, xs, dys, stats, g4[0], g4[1]):
        bn.backward_stage1(x, dy, st[:C], st[C:], scale, b[:C], b[C:], a[:C], a[C:])
    emu.allreduce_all(bes, g4[0])
    emu.allreduce_all(bes, g4[1])
    for bn, x, dy, dx, st, a in zip(bns, xs, dys, dxs, stats, g4[0]):
        bn.backward_stage2(x, dy, st[:C], st[C:], scale, a[:C], a[C:], dx)
    m_g, v_g = stats[0][:C].cpu().numpy(), stats[0][C:].cpu().numpy()
    dsc, dbi, dme, dva = O.bn_backprop1(g, gdy, m_g, v_g, scale.cpu().numpy(), 1e-5)
    emu.assert_close(g4[1][0][:C].cpu().numpy(), dsc, 2e-5, "dscale")
    emu.assert_close(g4[1][0][C:].cpu().numpy(), dbi, 2e-5, "dbias")
    dx_ref = O.bn_backprop2(g, gdy, m_g, v_g, scale.cpu().numpy(), g4[0][0][:C].cpu().numpy(),
                            g4[0][0][C:].cpu().numpy(), 1e-5, nps)
    emu.assert_close(emu.gather_owned(dxs, g.shape), dx_ref, 1e-5, "dx")


def test_leaky_relu():
    shape = [33, 9, 4, 2]
    be = dc.BackendDNNLib(dc.Locale(0, 1))
    x_t, y_t, dy_t, dx_t = (_rank0(shape, [1] * 4, [0] * 4) for _ in range(4))
    rng = np.random.default_rng(0)
    x = rng.normal(size=x_t.np_real_shape()).astype(np.float32)
    dy = rng.normal(size=x.shape).astype(np.float32)
    emu.upload(x_t, x)
    emu.upload(dy_t, dy)
    y_t.allocate()
    dx_t.allocate()
    lr = dc.LeakyReLU(be)
    lr.forward(x_t, 0.01, y_t)
    lr.backward(x_t, dy_t, 0.01, dx_t)
    assert np.array_equal(y_t.buffer.cpu().numpy(), np.where(x > 0, x, np.float32(0.01) * x))
    assert np.array_equal(dx_t.buffer.cpu().numpy(), np.where(x > 0, dy, np.float32(0.01) * dy))


def test_bn_apply_fused_with_leaky_relu_matches_the_two_passes():
    rng = np.random.default_rng(3)
    x = torch.from_numpy(rng.normal(0.1, 1.5, (2, 5, 6, 7, 40)).astype(np.float32)).cuda()
    C = 5
    mean = torch.from_numpy(rng.normal(0, 0.3, C).astype(np.float32)).cuda()
    var = torch.from_numpy(rng.uniform(0.5, 2, C).astype(np.float32)).cuda()
    scale = torch.from_numpy(rng.uniform(0.5, 1.5, C).astype(np.float32)).cuda()
    bias = torch.from_numpy(rng.normal(0, 0.5, C).astype(np.float32)).cuda()
    loc = dc.Locale(0, 1)
    be = dc.BackendDNNLib(loc, allreduce="peer", allreduce_max_count=64)
    shape = [40, 7, 6, C, 2]
    dist = dc.Distribution.make_localized_distribution(5)
    tx, ty, tz, tf = (dc.Tensor(shape, loc, dist) for _ in range(4))
    for t in (tx, ty, tz, tf):
        t.allocate()
    tx.buffer.copy_(x)
    bn = dc.BatchNormalization(be, 5, 0.9, 1e-5, True)
    rm, rv = torch.zeros(C, device="cuda"), torch.ones(C, device="cuda")
    bn.forward_stage2(tx, mean, var, rm, rv, scale, bias, ty, is_training=False)
    dc.LeakyReLU(be).forward(ty, 0.01, tz)
    bn.forward_stage2(tx, mean, var, rm, rv, scale, bias, tf, is_training=False, leaky_relu_slope=0.01)
    torch.cuda.synchronize()
    assert torch.equal(tf.buffer, tz.buffer)


def test_empty_shard_zero_fills_run_on_the_backend_stream():
    """A rank without cells contributes zeros to the all-reduces; those fills
    must be ordered on the backend's stream like the kernels they replace.
    The stream is kept busy, then writes 5s: a fill on another stream would
    run first and the 5s would survive."""
    side = torch.cuda.Stream()
    locale = dc.Locale(1, 2)
    be = dc.BackendDNNLib(locale, stream=side, connect=False)
    # D extent 1 over two ranks: the second one owns nothing
    t = dc.Tensor([8, 8, 1, 4, 1], locale, dc.Distribution.make_overlapped_distribution([1, 1, 2, 1, 1], [0] * 5))
    assert t.get_local_size() == 0
    t.allocate()
    bn = dc.BatchNormalization(be, 5, 0.9, 1e-5, True)
    vals = [torch.ones(4, device="cuda") for _ in range(6)]
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)
        for v in vals:
            v.fill_(5.0)
    bn.forward_stage1(t, vals[0], vals[1], True)
    bn.backward_stage1(t, t, vals[0], vals[1], vals[0], vals[2], vals[3], vals[4], vals[5])
    torch.cuda.synchronize()
    for v in vals:
        assert float(v.abs().max()) == 0.0


def _bn_problem(C=6, w=40):
    """A layer whose statistics come with its convolution: sums in, normalised output out."""
    gen = torch.Generator(device="cuda").manual_seed(2)
    be = dc.BackendDNNLib(dc.Locale(0, 1))
    x, y = (dc.Tensor([w, 9, 7, C, 2], dc.Locale(0, 1), dc.Distribution.make_localized_distribution(5)) for _ in range(2))
    for t in (x, y):
        t.allocate()
    x.buffer.copy_(torch.randn(x.buffer.shape, device="cuda", generator=gen) + 0.3)
    sums = torch.cat([x.owned().double().sum((0, 2, 3, 4)), x.owned().double().square().sum((0, 2, 3, 4))]).float()
    rest = [torch.zeros(C, device="cuda"), torch.ones(C, device="cuda"), torch.rand(C, device="cuda") + 0.5,
            torch.randn(C, device="cuda")]
    return be, x, y, sums, rest


def test_forward_on_given_statistics_needs_no_call_before_a_capture():
    """The first forward pass of a batch-norm whose sums are given may be a captured
    one: it allocates nothing."""
    be, x, y, sums, (rm, rv, scale, bias) = _bn_problem()
    C = sums.numel() // 2
    stats, bn = sums.clone(), dc.BatchNormalization(be, 5, 0.9, 1e-5, True)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        stats.copy_(sums)
        bn.forward(x, stats[:C], stats[C:], rm, rv, scale, bias, y, True, statistics_ready=True)
    rm.zero_(), rv.fill_(1.0)
    graph.replay()
    torch.cuda.synchronize()
    mean, var = x.owned().double().mean((0, 2, 3, 4)), x.owned().double().var((0, 2, 3, 4))
    assert torch.allclose(stats[:C].double(), mean, atol=1e-6) and torch.allclose(stats[C:].double(), var, rtol=1e-5)
    assert torch.allclose(rm.double(), 0.1 * mean, atol=1e-6)
    sh = (1, C, 1, 1, 1)
    ref = (x.owned().double() - mean.view(sh)) * (var.view(sh) + 1e-5).rsqrt() * scale.double().view(sh) + bias.double().view(sh)
    assert torch.allclose(y.owned().double(), ref, atol=2e-5)


def test_forward_passes_of_one_object_on_several_streams():
    """forward_stage2 keeps nothing between calls: passes of one object over different
    batches may run side by side, as separate finalize and apply calls may."""
    be, x, _, sums, (_, _, scale, bias) = _bn_problem(C=16, w=64)
    C, bn = 16, dc.BatchNormalization(be, 5, 0.9, 1e-5, True)
    streams, outs = [torch.cuda.Stream() for _ in range(4)], []
    for _ in range(8):
        y = dc.Tensor(x.shape, x.locale, x.dist)
        y.allocate()
        outs.append((y, sums.clone(), torch.zeros(C, device="cuda"), torch.ones(C, device="cuda")))
    torch.cuda.synchronize()
    for rep in range(20):
        for i, (y, st, rm, rv) in enumerate(outs):
            with torch.cuda.stream(streams[i % 4]):
                st.copy_(sums), rm.zero_(), rv.fill_(1.0)
                be.stream = streams[i % 4]
                bn.forward_stage2(x, st[:C], st[C:], rm, rv, scale, bias, y, True)
        torch.cuda.synchronize()
        for y, st, rm, rv in outs[1:]:
            assert torch.equal(st, outs[0][1]) and torch.equal(rm, outs[0][2]) and torch.equal(rv, outs[0][3])
            assert torch.equal(y.buffer, outs[0][0].buffer)
        assert not torch.equal(outs[0][1], sums)


def test_one_object_on_tensors_of_one_shape_and_several_pitches():
    """The kernels read x through the plan's strides."""
    be, x, y, sums, (rm, rv, scale, bias) = _bn_problem(C=4, w=33)
    C, bn = 4, dc.BatchNormalization(be, 5, 0.9, 1e-5, True)
    padded = dc.Tensor(x.shape, x.locale, x.dist, pitch_align=8)
    padded.allocate()
    padded.buffer.fill_(float("nan"))
    padded.owned().copy_(x.owned())
    assert padded.pitch != x.pitch and padded.get_local_shape() == x.get_local_shape()
    for t in (x, padded, x):
        st = torch.zeros(2 * C, device="cuda")
        bn.forward_stage1(t, st[:C], st[C:], True)
        assert torch.allclose(st, sums, rtol=1e-5, atol=1e-3)
        grads = [torch.zeros(C, device="cuda") for _ in range(4)]
        bn.backward_stage1(t, x, rm, rv, scale, *grads)
        assert torch.allclose(grads[1], sums[:C], rtol=1e-5, atol=1e-3)  # dbias: the sum of dy
