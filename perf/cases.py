"""The work that this library's callers have it do, as cases that can be timed.

A case is one step of a spatially parallel network through the operators of
``dihydrogen_b200``:

* ``layer``    convolution + batch-norm: ``fwd`` is the forward half of a training
               step (statistics, running statistics), ``train`` a forward and a
               backward pass (dx, dw, dscale, dbias), ``infer`` the forward pass on
               running statistics with the LeakyReLU that follows it
* ``pool``     pooling of an activation, forward and backward
* ``halo``     one halo exchange of a partitioned tensor
* ``shuffle``  a re-distribution from sample-parallel to spatially partitioned and
               the one back

Where ``ranks`` is 2, both ranks' shards live in this process, on one GPU, and every
phase is called for both before the next one, so that no call waits for a later
one.  Extents are those of the whole tensor; ``split`` is the partitioned dimension
(0 is W).  Tensors are single precision; ``math`` is the precision that the
convolution's forward and backward-data products are taken in.
"""
import math

import torch

import dihydrogen_b200 as dc
from dihydrogen_b200 import _abi

DECAY, EPS, SLOPE = 0.9, 1e-5, 0.01
MATH = {"fp32": _abi.MATH_FP32, "tf32": _abi.MATH_TF32, "bf16": _abi.MATH_BF16}


def _layer(name, do, n, c, k, d, h, w, f, stride=1, math="fp32", ranks=1, split=0):
    """d == 0: a 2-D layer."""
    case = {"kind": "layer", "do": do, "n": n, "c": c, "k": k, "d": d, "h": h, "w": w, "f": f, "stride": stride,
            "math": math, "ranks": ranks, "split": split}
    return dict(case, name=name) if name else case


def listed():
    return [
        # the 2-D layer of the reference's CPU example: small images, where launches and host time count
        _layer("layer2d_64_fwd", "fwd", 4, 16, 16, 0, 64, 64, 3),
        # a deep, small volume late in a network: a whole training step of a few hundred kilobytes
        _layer("layer3d_32_train", "train", 1, 4, 16, 16, 24, 32, 3),
        # the first layer of a CosmoFlow-style network on one GPU's shard: forward, and the training step
        _layer("layer3d_256_fwd", "fwd", 1, 4, 16, 256, 256, 256, 3),
        _layer("layer3d_256_train", "train", 1, 4, 16, 256, 256, 256, 3),
        # its second layer, which halves the volume
        _layer("layer3d_256_s2_train", "train", 1, 16, 32, 256, 256, 256, 3, stride=2),
        # segmentation of large images: wide 5 x 5 filters on one GPU's shard of a 4096 x 4096 pair
        _layer("layer2d_2048_f5_train", "train", 2, 32, 32, 0, 2048, 1024, 5),
        # a cropped volume: no extent is a multiple of anything, two samples
        _layer("layer3d_ragged_train", "train", 2, 8, 24, 67, 83, 101, 3),
        # serving a trained network at reduced precision
        _layer("layer3d_128_infer_bf16", "infer", 1, 4, 16, 128, 128, 128, 3, math="bf16"),
        # a volume cut in two along W: halos in both passes, padded rows
        _layer("layer3d_split_w_train", "train", 1, 4, 16, 128, 128, 256, 3, ranks=2, split=0),
        # max-pooling of the first layer's output, both directions
        {"name": "pool3d_256", "kind": "pool", "n": 1, "c": 16, "d": 256, "h": 256, "w": 256, "window": 3, "stride": 2,
         "pad": 1, "mode": "MAX"},
        # the halo of the first layer's output when the volume is cut along W, the most scattered of the faces
        {"name": "halo_256_w", "kind": "halo", "c": 16, "d": 256, "h": 256, "w": 256, "width": 1, "split": 0, "ranks": 2},
        # from whole samples per rank to volumes cut along D and back
        {"name": "shuffle_128", "kind": "shuffle", "n": 2, "c": 16, "d": 128, "h": 128, "w": 128, "split": 2, "ranks": 2},
    ]


def _extent(rng, lo, hi):
    """Spread over the logarithm; half of them even multiples of 8, the rest as they fall."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, v // 8 * 8) if rng.random() < 0.5 else v


def draw(rng):
    kind = rng.choice(["layer"] * 7 + ["pool", "halo", "shuffle"])
    while True:
        if kind == "layer":
            flat = rng.random() < 0.35
            d = 0 if flat else _extent(rng, 16, 256)
            h, w = (_extent(rng, 32, 2048), _extent(rng, 32, 2048)) if flat else (_extent(rng, 16, 256), _extent(rng, 16, 256))
            case = _layer(None, rng.choice(["fwd", "train", "train", "infer"]), rng.choice([1, 1, 2, 4]),
                          _extent(rng, 1, 32), _extent(rng, 4, 32), d, h, w, rng.choice([3, 5]) if flat else 3,
                          stride=rng.choice([1, 1, 1, 2]), math=rng.choice(["fp32", "fp32", "fp32", "tf32", "bf16"]))
            if case["stride"] == 1 and case["math"] == "fp32" and rng.random() < 0.25:
                case.update(ranks=2, split=rng.randrange(2 if flat else 3))
        elif kind == "pool":
            window, stride, pad = rng.choice([(3, 2, 1), (3, 2, 1), (2, 2, 0), (3, 1, 1)])
            case = {"kind": "pool", "n": rng.choice([1, 1, 2]), "c": rng.choice([4, 8, 16, 32]), "d": _extent(rng, 16, 256),
                    "h": _extent(rng, 16, 256), "w": _extent(rng, 16, 256), "window": window, "stride": stride, "pad": pad,
                    "mode": rng.choice(["MAX", "MAX", "AVERAGE"])}
        else:
            case = {"kind": kind, "c": rng.choice([4, 8, 16, 32, 64]), "d": _extent(rng, 32, 256), "h": _extent(rng, 32, 256),
                    "w": _extent(rng, 32, 256), "split": rng.randrange(3), "ranks": 2}
            case.update({"width": rng.choice([1, 1, 2, 3])} if kind == "halo" else {"n": 2})
        todo = work(case)
        # within the listed ones' cost, and large enough to be a case at all
        if todo["flops"] <= 1.5e11 and 2e5 <= todo["bytes"] <= 1.5e9 and _held(case) <= 4e9:
            return case


# -- sizes ---------------------------------------------------------------------
def _spatial(case):
    """Extents of the input, W first."""
    return [case["w"], case["h"]] + ([case["d"]] if case["d"] else [])


def _filter(case):
    return [case["f"]] * len(_spatial(case))


def _out(case, f, stride, pad):
    return [(e + 2 * pad - f) // stride + 1 for e in _spatial(case)]


def _cells(case):
    """Values in the input and in the output of a layer or a pooling."""
    if case["kind"] == "layer":
        out = _out(case, case["f"], case["stride"], (case["f"] - 1) // 2)
        return (case["n"] * case["c"] * math.prod(_spatial(case)), case["n"] * case["k"] * math.prod(out))
    out = _out(case, case["window"], case["stride"], case["pad"])
    return case["n"] * case["c"] * math.prod(_spatial(case)), case["n"] * case["c"] * math.prod(out)


def _held(case):
    """Bytes that a state holds on the device, about."""
    if case["kind"] in ("layer", "pool"):
        a, b = _cells(case)
        return 4 * (2 * a + 4 * b)
    return 4 * case.get("n", 1) * case["c"] * math.prod(_spatial(case)) * 4


def work(case):
    if case["kind"] == "layer":
        x, y = _cells(case)
        taps = case["c"] * math.prod(_filter(case))
        macs = y * taps
        if case["do"] == "infer":
            return {"bytes": 4 * (x + y), "flops": 2 * macs + 2 * y}
        if case["do"] == "fwd":  # the convolution's output and the normalised one
            return {"bytes": 4 * (x + 2 * y), "flops": 2 * macs + 6 * y}
        return {"bytes": 4 * (2 * x + 3 * y + 2 * case["k"] * taps), "flops": 6 * macs + 20 * y}
    if case["kind"] == "pool":
        x, y = _cells(case)
        return {"bytes": 4 * (2 * x + 2 * y), "flops": 2 * y * case["window"] ** 3}
    sp = _spatial(case)
    if case["kind"] == "halo":  # two faces, each read and written into the neighbour's halo cells
        face = case["width"] * case["c"] * math.prod(e for i, e in enumerate(sp) if i != case["split"])
        return {"bytes": 2 * 8 * face, "flops": 0}
    return {"bytes": 2 * 8 * case["n"] * case["c"] * math.prod(sp), "flops": 0}


def tolerance(case):
    if case["kind"] in ("halo", "shuffle"):
        return "exact"
    if case["kind"] == "pool":
        return {"rel": 1e-6}
    return {"rel": {"fp32": 1e-5, "tf32": 1e-3, "bf16": 1e-2}[case["math"]]}


# -- states --------------------------------------------------------------------
def _randn(gen, shape):
    return torch.randn(shape, generator=gen, device="cuda")


def _fill(gen, tensor, activation):
    """The owned cells: what a LeakyReLU passes on, or a gradient."""
    own = tensor.owned()
    v = _randn(gen, tuple(own.shape))
    own.copy_(torch.where(v < 0, SLOPE * v, v) if activation else 1e-2 * v)


def _connect(exchangers):
    blobs = [e.export() for e in exchangers]
    for e in exchangers:
        e.connect(blobs)


def _prepare_layer(case, gen):
    sp, f = _spatial(case), _filter(case)
    nsd, ranks, k, c = len(sp), case["ranks"], case["k"], case["c"]
    grid = [1] * (nsd + 2)
    grid[case["split"]] = ranks
    strides, dil, pads = [case["stride"]] * nsd, [1] * nsd, [(e - 1) // 2 for e in f]
    train = case["do"] == "train"
    filt = _randn(gen, (k, c, *f)) * math.sqrt(2.0 / (c * math.prod(f)))  # all extents are equal: no order to reverse
    scale, bias = 1 + 0.1 * _randn(gen, (k,)), 0.1 * _randn(gen, (k,))
    shards = []
    for rank in range(ranks):
        locale = dc.Locale(rank, ranks)
        s = {"x": dc.create_input_tensor(sp + [c, case["n"]], grid, f, strides, dil, locale)}
        s["y"] = dc.create_convolution_output_tensor(s["x"], f + [c, k], strides, pads, dil)
        s["z"] = dc.Tensor(s["y"].shape, locale, s["y"].dist, s["y"]._local_of)
        if train:
            s["dx"] = dc.create_d_input_tensor(s["x"])
            s["dy"] = dc.create_convolution_d_output_tensor(s["y"], f + [c, k], dil)
            s["dz"] = dc.Tensor(s["y"].shape, locale, s["y"].dist, s["y"]._local_of)
        for t in s.values():
            t.allocate()
        _fill(gen, s["x"], True)
        be = dc.BackendDNNLib(locale, options=dc.Options(math_mode=MATH[case["math"]]), connect=ranks == 1)
        conv = dc.Convolution(be, nsd + 2)
        s["dw"] = torch.zeros_like(filt) if train else None
        conv.setup(s["x"], filt, s["y"], s.get("dx"), s["dw"], s.get("dy"), pads, strides, dil, connect=ranks == 1)
        if train:
            _fill(gen, s["dz"], False)
        s.update(be=be, conv=conv, bn=dc.BatchNormalization(be, nsd + 2, DECAY, EPS, True),
                 stats=torch.zeros(2 * k, device="cuda"), grads=torch.zeros(4 * k, device="cuda"),
                 running_mean=torch.full((k,), 0.1, device="cuda"), running_var=torch.ones(k, device="cuda"))
        shards.append(s)
    if ranks > 1:
        _connect([s["be"].allreducer for s in shards])
        _connect([s["conv"].halo_xch_input for s in shards])
        if train:
            _connect([s["conv"].halo_xch_d_output for s in shards])
    return {"case": case, "shards": shards, "filter": filt, "scale": scale, "bias": bias}


def _prepare_pool(case, gen):
    sp = _spatial(case)
    nsd, locale = len(sp), dc.Locale(0, 1)
    window, strides, pads = [case["window"]] * nsd, [case["stride"]] * nsd, [case["pad"]] * nsd
    x = dc.create_input_tensor(sp + [case["c"], case["n"]], [1] * (nsd + 2), window, strides, [1] * nsd, locale)
    y = dc.create_pooling_output_tensor(x, window, strides, pads)
    dx, dy = dc.create_d_input_tensor(x), dc.create_pooling_d_output_tensor(y)
    for t in (x, y, dx, dy):
        t.allocate()
    _fill(gen, x, True)
    _fill(gen, dy, False)
    pool = dc.Pooling(dc.BackendDNNLib(locale), nsd + 2)
    pool.setup(x, y, dx, dy, window, pads, strides, case["mode"])
    return {"case": case, "x": x, "y": y, "dx": dx, "dy": dy, "pool": pool}


def _prepare_halo(case, gen):
    sp = _spatial(case)
    grid, overlap = [1] * (len(sp) + 2), [0] * (len(sp) + 2)
    grid[case["split"]], overlap[case["split"]] = case["ranks"], case["width"]
    tensors = []
    for rank in range(case["ranks"]):
        t = dc.Tensor(sp + [case["c"], 1], dc.Locale(rank, case["ranks"]),
                      dc.Distribution.make_overlapped_distribution(grid, overlap))
        t.allocate()
        _fill(gen, t, True)
        tensors.append(t)
    exchangers = [dc.HaloExchange(t) for t in tensors]
    _connect(exchangers)
    return {"case": case, "tensors": tensors, "exchangers": exchangers}


def _prepare_shuffle(case, gen):
    sp = _spatial(case)
    by_sample, by_volume = [1] * (len(sp) + 2), [1] * (len(sp) + 2)
    by_sample[-1], by_volume[case["split"]] = case["ranks"], case["ranks"]
    shards = []
    for rank in range(case["ranks"]):
        locale = dc.Locale(rank, case["ranks"])
        src, dst, back = (dc.Tensor(sp + [case["c"], case["n"]], locale, dc.Distribution.make_distribution(g))
                          for g in (by_sample, by_volume, by_sample))
        for t in (src, dst, back):
            t.allocate()
        _fill(gen, src, True)
        shards.append({"src": src, "dst": dst, "back": back, "shuffler": dc.TensorShuffler(src, dst, connect=False)})
    for which in ("fwd", "bwd"):
        blobs = [s["shuffler"].export(which) for s in shards]
        for s in shards:
            s["shuffler"].connect(which, blobs)
    return {"case": case, "shards": shards}


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    return {"layer": _prepare_layer, "pool": _prepare_pool, "halo": _prepare_halo, "shuffle": _prepare_shuffle}[case["kind"]](case, gen)


# -- passes --------------------------------------------------------------------
def _exchange(exchangers, dim, **how):
    for e in exchangers:
        e.pack_put(dim, **how)
    for e in exchangers:
        e.wait_unpack(dim)


def _sum_over_ranks(shards, vectors):
    for s, v in zip(shards, vectors):
        s["be"].allreducer.push(v.data_ptr(), v.numel())
    for s, v in zip(shards, vectors):
        s["be"].allreducer.pull(v.data_ptr(), v.numel())


def _run_layer(st):
    case, filt, k = st["case"], st["filter"], st["case"]["k"]
    if case["ranks"] > 1:
        return _run_layer_ranks(st)
    s = st["shards"][0]
    conv, bn, x, y, z = s["conv"], s["bn"], s["x"], s["y"], s["z"]
    mean, var, rm, rv = s["stats"][:k], s["stats"][k:], s["running_mean"], s["running_var"]
    if case["do"] == "infer":
        conv.forward(1.0, x, filt, 0.0, y, inference=True)
        bn.forward_stage2(y, mean, var, rm, rv, st["scale"], st["bias"], z, False, leaky_relu_slope=SLOPE)
        return [z.owned()]
    ready = conv.forward(1.0, x, filt, 0.0, y, statistics=(mean, var)) == 1
    bn.forward(y, mean, var, rm, rv, st["scale"], st["bias"], z, True, statistics_ready=ready)
    out = [y.owned(), z.owned(), rm, rv]
    if case["do"] == "train":
        dscale, dbias, dmean, dvar = s["grads"].split(k)
        bn.backward(y, s["dz"], mean, var, st["scale"], dscale, dbias, dmean, dvar, s["dy"])
        conv.backward_filter(1.0, x, s["dy"], 0.0, s["dw"])
        conv.backward_data(1.0, filt, s["dy"], 0.0, s["dx"])
        out += [s["dx"].owned(), s["dw"], dscale, dbias]
    return out


def _run_layer_ranks(st):
    case, shards, filt, k = st["case"], st["shards"], st["filter"], st["case"]["k"]
    dim, train = case["split"], case["do"] == "train"
    _exchange([s["conv"].halo_xch_input for s in shards], dim, clear_boundary=True)
    if case["do"] == "infer":
        for s in shards:
            s["conv"].forward(1.0, s["x"], filt, 0.0, s["y"], skip_halo_exchange=True, inference=True)
            s["bn"].forward_stage2(s["y"], s["stats"][:k], s["stats"][k:], s["running_mean"], s["running_var"], st["scale"],
                                   st["bias"], s["z"], False, leaky_relu_slope=SLOPE)
        return [s["z"].owned() for s in shards]
    for s in shards:
        mean, var = s["stats"][:k], s["stats"][k:]
        if not s["conv"].forward(1.0, s["x"], filt, 0.0, s["y"], skip_halo_exchange=True, statistics=(mean, var)):
            s["bn"].forward_stage1(s["y"], mean, var, True)
    _sum_over_ranks(shards, [s["stats"] for s in shards])
    out = []
    for s in shards:
        s["bn"].forward_stage2(s["y"], s["stats"][:k], s["stats"][k:], s["running_mean"], s["running_var"], st["scale"],
                               st["bias"], s["z"], True)
        out += [s["y"].owned(), s["z"].owned(), s["running_mean"], s["running_var"]]
    if not train:
        return out
    for s in shards:
        s["bn"].backward_stage1(s["y"], s["dz"], s["stats"][:k], s["stats"][k:], st["scale"], *s["grads"].split(k))
    _sum_over_ranks(shards, [s["grads"] for s in shards])
    for s in shards:
        dscale, dbias, dmean, dvar = s["grads"].split(k)
        s["bn"].backward_stage2(s["y"], s["dz"], s["stats"][:k], s["stats"][k:], st["scale"], dmean, dvar, s["dy"])
        s["conv"].backward_filter(1.0, s["x"], s["dy"], 0.0, s["dw"], reduce=False)
        out += [dscale, dbias]
    _sum_over_ranks(shards, [s["dw"] for s in shards])
    _exchange([s["conv"].halo_xch_d_output for s in shards], dim, clear_boundary=True)
    for s in shards:
        s["conv"].backward_data(1.0, filt, s["dy"], 0.0, s["dx"], skip_halo_exchange=True)
        out += [s["dx"].owned(), s["dw"]]
    return out


def _run_pool(st):
    st["pool"].forward(1.0, st["x"], 0.0, st["y"])
    st["pool"].backward(1.0, st["y"], st["dy"], st["x"], 0.0, st["dx"])
    return [st["y"].owned(), st["dx"].owned()]


def _run_halo(st):
    _exchange(st["exchangers"], st["case"]["split"])
    return [t.buffer for t in st["tensors"]]


def _run_shuffle(st):
    for which, src, dst in (("fwd", "src", "dst"), ("bwd", "dst", "back")):
        for s in st["shards"]:
            s["shuffler"].put(which, s[src].get_buffer())
        for s in st["shards"]:
            s["shuffler"].wait_unpack(which, s[dst].get_buffer())
    return [s[t].owned() for s in st["shards"] for t in ("dst", "back")]


def run(state):
    return {"layer": _run_layer, "pool": _run_pool, "halo": _run_halo, "shuffle": _run_shuffle}[state["case"]["kind"]](state)
