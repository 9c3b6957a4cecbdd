"""Re-distribution between two block decompositions on emulated ranks: every
cell ends up with its owner in the other distribution (bit-exact), halo cells
of the destination are left alone, and the way back restores the source."""
import numpy as np
import pytest
import torch

import dihydrogen_b200 as dc
from dihydrogen_b200 import _abi

import emu

pytestmark = pytest.mark.gpu

# global shape (W, H, [D,] C, N), source grid, destination grid, destination overlap
CASES = [
    ([12, 10, 8, 3, 4], [1, 1, 1, 1, 4], [1, 1, 4, 1, 1], [0, 0, 1, 0, 0]),   # sample-parallel -> D-partitioned with halo
    ([12, 10, 8, 3, 4], [2, 2, 1, 1, 1], [1, 1, 2, 1, 2], [0, 0, 1, 0, 0]),   # 2x2 in W, H -> D x N
    ([20, 9, 2, 6], [1, 3, 1, 2], [2, 1, 1, 3], [1, 0, 0, 0]),                # 4-D, ragged splits, 6 ranks
    ([16, 8, 8, 2, 1], [1, 1, 1, 1, 1], [1, 1, 1, 1, 1], [0, 0, 0, 0, 0]),    # one rank: a local copy
    ([7, 5, 3, 2, 2], [1, 1, 3, 1, 1], [1, 1, 3, 1, 1], [0, 0, 1, 0, 0]),     # same split, only the halo differs
]


def _tensor(shape, grid, overlap, loc):
    return dc.Tensor(shape, loc, dc.Distribution.make_overlapped_distribution(grid, overlap))


@pytest.mark.parametrize("shape,sgrid,dgrid,dov", CASES)
def test_forward_and_backward(shape, sgrid, dgrid, dov):
    n = int(np.prod(sgrid))
    assert n == int(np.prod(dgrid))
    rng = np.random.default_rng(1)
    g = rng.normal(size=tuple(reversed(shape))).astype(np.float32)
    srcs, dsts, backs, shufflers = [], [], [], []
    for loc in emu.locales(n):
        s = _tensor(shape, sgrid, [0] * len(shape), loc)
        d = _tensor(shape, dgrid, dov, loc)
        b = _tensor(shape, sgrid, [0] * len(shape), loc)
        emu.scatter_owned(s, g)
        d.allocate()
        d.buffer.fill_(-7.0)
        b.allocate()
        srcs.append(s), dsts.append(d), backs.append(b)
        shufflers.append(dc.TensorShuffler(s, d, connect=False))
    for which in ("fwd", "bwd"):
        blobs = [sh.export(which) for sh in shufflers]
        for sh in shufflers:
            sh.connect(which, blobs)
    for rep in range(3):  # the receive windows alternate: run through both halves
        for sh, s in zip(shufflers, srcs):
            sh.put("fwd", s.get_buffer())
        for sh, d in zip(shufflers, dsts):
            sh.wait_unpack("fwd", d.get_buffer())
    torch.cuda.synchronize()
    assert np.array_equal(emu.gather_owned(dsts, g.shape), g)
    for d in dsts:  # halo cells untouched
        own = torch.zeros_like(d.buffer, dtype=torch.bool)
        own[tuple(slice(o, o + l) for o, l in reversed(list(zip(d.dist.overlap, d.local_shape))))] = True
        assert bool((d.buffer[~own] == -7.0).all())
    for sh, d in zip(shufflers, dsts):
        sh.put("bwd", d.get_buffer())
    for sh, b in zip(shufflers, backs):
        sh.wait_unpack("bwd", b.get_buffer())
    torch.cuda.synchronize()
    assert np.array_equal(emu.gather_owned(backs, g.shape), g)
    assert all(sh.status("fwd") == _abi.OK and sh.status("bwd") == _abi.OK for sh in shufflers)


@pytest.mark.parametrize("shape,sgrid,dgrid,dov", [
    # runs of 5 and 6 cells: cell by cell and, from 6 on, in pieces
    ([11, 5, 4, 3, 2], [1, 1, 1, 1, 2], [2, 1, 1, 1, 1], [0, 0, 0, 0, 0]),
    # ... with a halo along W, where rows start 1 to 3 cells off a boundary
    ([13, 6, 4, 2, 2], [1, 1, 1, 1, 2], [2, 1, 1, 1, 1], [1, 0, 0, 0, 0]),
    ([14, 6, 4, 2, 2], [1, 1, 1, 1, 2], [2, 1, 1, 1, 1], [2, 1, 0, 0, 0]),
    # merged rows of odd length, split in H
    ([13, 11, 9, 3, 2], [1, 1, 1, 1, 2], [1, 2, 1, 1, 1], [0, 0, 0, 0, 0]),
    ([10, 9, 5, 3, 2], [1, 1, 1, 1, 2], [1, 2, 1, 1, 1], [0, 1, 0, 0, 0]),
    # runs of 2070 and 4092 cells, below and at the 1024 pieces from which a run has its own units
    ([45, 92, 3, 3, 2], [1, 1, 1, 1, 2], [1, 2, 1, 1, 1], [0, 0, 0, 0, 0]),
    ([62, 132, 3, 2, 2], [1, 1, 1, 1, 2], [1, 2, 1, 1, 1], [0, 1, 0, 0, 0]),
    ([45, 182, 3, 2, 2], [1, 1, 1, 1, 2], [1, 2, 1, 1, 1], [0, 0, 0, 0, 0]),
    # whole odd planes: runs of several units, in pieces
    ([97, 91, 3, 2, 2], [1, 1, 1, 1, 2], [1, 1, 2, 1, 1], [0, 0, 0, 0, 0]),
    ([98, 91, 3, 1, 2], [1, 1, 1, 1, 2], [1, 1, 2, 1, 1], [0, 0, 1, 0, 0]),
])
def test_runs_off_16_byte_boundaries(shape, sgrid, dgrid, dov):
    test_forward_and_backward(shape, sgrid, dgrid, dov)


@pytest.mark.parametrize("shape,dgrid,dov", [
    ([128, 128, 104, 8, 2], [1, 1, 2, 1, 1], [0, 0, 1, 0, 0]),   # whole planes: 16-byte accesses, jobs of several units
    ([10, 127, 128, 84, 2], [2, 1, 1, 1, 1], [0, 0, 0, 0, 0]),   # runs of 5 cells, one by one; the last unit is short
    ([8, 130, 126, 105, 2], [2, 1, 1, 1, 1], [1, 0, 0, 0, 0]),   # of 4, rows off a boundary by the halo
])
def test_large_windows(shape, dgrid, dov):
    """Unpacked from their end (no pieces in them)."""
    assert 4 * np.prod(shape) >= 0.75 * torch.cuda.get_device_properties(0).L2_cache_size
    test_forward_and_backward(shape, [1, 1, 1, 1, 2], dgrid, dov)


@pytest.mark.parametrize("src_off,dst_off", [(1, 0), (0, 2), (3, 1)])
@pytest.mark.parametrize("shape,dgrid,dov", [
    ([16, 8, 4, 3, 2], [2, 1, 1, 1, 1], [0, 0, 0, 0, 0]),     # runs of 8 cells
    ([8, 8, 4, 3, 2], [2, 1, 1, 1, 1], [0, 0, 0, 0, 0]),      # of 4: cell by cell
    ([24, 20, 6, 3, 2], [1, 2, 1, 1, 1], [0, 1, 0, 0, 0]),    # rows merged
    ([64, 72, 6, 2, 2], [1, 1, 2, 1, 1], [0, 0, 1, 0, 0]),    # long runs
])
def test_tensors_off_16_byte_boundaries(shape, dgrid, dov, src_off, dst_off):
    """Everything is a multiple of 16 bytes but the tensors' own addresses: 16-byte accesses are out, pieces are not."""
    sgrid, g = [1, 1, 1, 1, 2], np.random.default_rng(2).normal(size=tuple(reversed(shape))).astype(np.float32)
    srcs, dsts, backs = ([_tensor(shape, grid, ov, loc) for loc in emu.locales(2)]
                         for grid, ov in ((sgrid, [0] * 5), (dgrid, dov), (sgrid, [0] * 5)))
    for ts, off in ((srcs, src_off), (dsts, dst_off), (backs, src_off)):
        for t in ts:
            emu.allocate_off_boundary(t, off)
            t.buffer.fill_(-7.0)
    for t in srcs:
        emu.scatter_owned_into(t, g)
    shufflers = [dc.TensorShuffler(s, d, connect=False) for s, d in zip(srcs, dsts)]
    for which, a, b in (("fwd", srcs, dsts), ("bwd", dsts, backs)):
        blobs = [sh.export(which) for sh in shufflers]
        for sh in shufflers:
            sh.connect(which, blobs)
        for sh, t in zip(shufflers, a):
            sh.put(which, t.get_buffer())
        for sh, t in zip(shufflers, b):
            sh.wait_unpack(which, t.get_buffer())
        torch.cuda.synchronize()
        assert np.array_equal(emu.gather_owned(b, g.shape), g)
        for t in b:  # halo cells untouched
            own = torch.zeros_like(t.buffer, dtype=torch.bool)
            own[t._geo().owned] = True
            assert bool((t.buffer[~own] == -7.0).all())
        assert all(sh.status(which) == _abi.OK for sh in shufflers)


def test_wait_expires_with_status_when_a_sender_never_comes():
    """A rank whose peer never puts gets DCB_PEER_TIMEOUT from the bounded wait,
    not a hang, and the destination stays as it was."""
    shape, n = [8, 6, 4, 2, 2], 2
    srcs, dsts, shufflers = [], [], []
    for loc in emu.locales(n):
        s = _tensor(shape, [1, 1, 1, 1, 2], [0] * 5, loc)
        d = _tensor(shape, [1, 1, 2, 1, 1], [0] * 5, loc)
        s.allocate(), d.allocate()
        srcs.append(s), dsts.append(d)
        shufflers.append(dc.TensorShuffler(s, d, connect=False))
    blobs = [sh.export("fwd") for sh in shufflers]
    for sh in shufflers:
        sh.connect("fwd", blobs)
    assert _abi.lib().dcb_set_wait_budget_ns(20_000_000) == _abi.OK
    try:
        shufflers[0].put("fwd", srcs[0].get_buffer())  # rank 1 never puts
        dsts[0].buffer.fill_(3.0)
        shufflers[0].wait_unpack("fwd", dsts[0].get_buffer())
        assert shufflers[0].status("fwd") == _abi.PEER_TIMEOUT
        assert bool((dsts[0].buffer == 3.0).all())
    finally:
        _abi.lib().dcb_set_wait_budget_ns(2_000_000_000)
