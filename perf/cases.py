"""The work that programs give this library, as cases that can be timed.

A network on sparse voxels calls it in four ways, and these are the kinds of case here:

* ``conv``   one submanifold convolution (K = 3).  Most layers get the neighbour cache of an earlier layer (``build``
             false: the cache is in the program's hands before the call); the first layer on an object builds it.
* ``stack``  residual blocks [conv, SiLU, conv] + skip on one cache that the first conv builds.
* ``down``   the strided ``sparse_conv3d`` between two levels: output coordinates, both maps and the convolution.
* ``sample`` ``grid_sample_3d``: features of the voxels read at arbitrary points near the surface.

``train`` runs the backward pass for all inputs that carry a gradient, otherwise the call is made under ``no_grad``.
The voxels are spherical shells (a surface at resolution ``res``, the geometry of ``flexgemm_b200.workloads``); an
object's place in the grid, its features, weights and gradients come from the seed.  Sizes follow the library's own
benchmark and tests: resolutions 8 to 1024, up to 8 objects, 16 to 1024 channels (wide at low resolution, narrow at
high), a few channels at the two ends of a network; fp16, bf16, fp32 as TF32 (the default) and fp32-accurate.
"""
import functools
import math
import random

import torch

from flexgemm_b200.kernels import config
from flexgemm_b200.ops.grid_sample import grid_sample_3d
from flexgemm_b200.ops.spconv import sparse_conv3d, sparse_submanifold_conv3d
from flexgemm_b200.workloads import shell_coords_torch

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32, "fp32_exact": torch.float32}
K = 3  # extent of the submanifold kernels


def _conv(name, **kw):
    return dict(dict(name=name, kind="conv", res=64, batch=1, ci=64, co=64, dtype="fp16", train=True, build=False, shuffled=False,
                     bias=True), **kw)


def listed():
    return [
        # a deep level of a small object at inference: the smallest call, all latency and launches
        _conv("deep_infer", res=16, ci=64, co=64, train=False),
        # the library's smoke test: a small fp32 layer trained
        _conv("small_train", res=32, ci=32, co=32, dtype="fp32"),
        # the wide bottom of a network: few voxels, 57 MB of weights
        _conv("wide_train", res=32, ci=1024, co=1024),
        # the headline benchmark: a large surface at a middle width
        _conv("surface_train", res=256, ci=256, co=256),
        # the sweep's fp32 point: TF32 at a large width
        _conv("tf32_train", res=128, ci=512, co=512, dtype="fp32"),
        # fp32 with accurate products, a few objects
        _conv("exact_train", res=64, batch=4, ci=128, co=128, dtype="fp32_exact"),
        # the first layer on a new object at inference: six input channels, the map is built
        _conv("first_infer", res=256, ci=6, co=64, train=False, build=True),
        # rows in no order (points as a loader delivers them), a channel count off the powers of two
        _conv("unordered_train", res=128, ci=96, co=96, dtype="bf16", build=True, shuffled=True),
        # two objects at the highest resolution, narrow: memory traffic, and the map of 5 M voxels
        _conv("hires_train", res=1024, batch=2, ci=64, co=64, build=True),
        # two blocks of the residual-stack benchmark
        dict(name="stack_train", kind="stack", res=64, batch=4, c=512, blocks=2, dtype="bf16", train=True),
        # between two levels: halving the resolution, doubling the width
        dict(name="down_train", kind="down", res=256, batch=1, ci=64, co=128, k=2, stride=2, pad=0, dtype="fp16", train=True),
        # a million surface points reading 256 channels
        dict(name="sample_train", kind="sample", res=256, batch=1, c=256, points=1_000_000, mode="trilinear", dtype="fp16", train=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw(rng):
    kind = rng.choices(("conv", "stack", "down", "sample"), (7, 1, 2, 2))[0]
    c = dict(kind=kind, res=_log(rng, 8, 1024), batch=rng.choice((1, 1, 1, 2, 3, 4, 8)),
             dtype=rng.choice(("fp16", "fp16", "fp16", "bf16", "bf16", "fp32", "fp32", "fp32_exact")), train=rng.random() < 0.7)
    width = 8 * max(2, _log(rng, 16, 1024) // 8)
    if kind == "conv":
        ends = rng.random()
        few = rng.randint(1, 12)
        c.update(ci=few if ends < 0.12 else width, co=few if ends > 0.94 else 8 * max(2, width // 16) if 0.12 < ends < 0.22 else width,
                 build=ends < 0.12 or rng.random() < 0.35, bias=rng.random() < 0.8)
        c["shuffled"] = c["build"] and rng.random() < 0.25
    elif kind == "stack":
        c.update(c=width, blocks=rng.randint(1, 4))
    elif kind == "down":
        c.update(ci=width, co=rng.choice((width, min(2 * width, 1024))))
        c.update(zip(("k", "stride", "pad"), rng.choice(((2, 2, 0), (3, 2, 1)))))
    else:
        c["dtype"] = c["dtype"].removesuffix("_exact")  # no products that TF32 would change
        c.update(c=width, points=_log(rng, 1_000, 2_000_000), mode=rng.choice(("trilinear", "trilinear", "nearest")))
    return c


def _cost(case):
    """Rough seconds of a pass, from closed forms (a shell has about 2.5 res^2 voxels and 10.5 pairs a voxel)."""
    n = 2.5 * case["res"] ** 2 * case["batch"]
    size = DTYPES[case["dtype"]].itemsize
    rate = {"fp16": 6e14, "bf16": 6e14, "fp32": 3e14, "fp32_exact": 1e14}[case["dtype"]]
    passes = 3 if case["train"] else 1
    if case["kind"] == "sample":
        return passes * case["points"] * case["c"] * size * (9 if case["mode"] == "trilinear" else 2) / 5e12
    ci, co = (case["c"], case["c"]) if case["kind"] == "stack" else (case["ci"], case["co"])
    convs = 2 * case.get("blocks", 0.5)
    return convs * passes * n * 10.5 * (2 * ci * co / rate + (ci + co) * size / 6e12)


_most = functools.lru_cache(None)(lambda: max(_cost(c) for c in listed()))


def draw(rng):
    while True:
        c = _draw(rng)
        if _cost(c) <= _most():
            return c


def _place(res, batch):
    return shell_coords_torch(res, batch, [1.0 - 0.2 * ((0.618 * b) % 1.0) for b in range(batch)],
                              device="cuda" if torch.cuda.is_available() else "cpu")


def _key(c, size):
    c = c.long()
    return ((c[:, 0] * size + c[:, 1]) * size + c[:, 2]) * size + c[:, 3]


@functools.lru_cache(None)
def _counts(res, batch, k, stride, pad):
    """(input rows, output rows, pairs) of a convolution on the shells of this size."""
    c = _place(res, batch)
    keys = _key(c, res)  # ascending: the rows are in lexicographic order
    pairs, outs = 0, []
    for v in range(k ** 3):
        d = torch.tensor([v // (k * k), v // k % k, v % k], device=c.device)
        if stride == 1:
            q = c[:, 1:] + d - k // 2
            ok = ((q >= 0) & (q < res)).all(1)
            want = _key(torch.cat([c[:, :1], q], 1), res)
            at = torch.searchsorted(keys, want).clamp_(max=max(len(keys) - 1, 0))
            pairs += int((ok & (keys[at] == want)).sum())
        else:
            size = (res + 2 * pad - k) // stride + 1
            q = c[:, 1:] + pad - d
            o = torch.div(q, stride, rounding_mode="floor")
            ok = ((q % stride == 0) & (o >= 0) & (o < size)).all(1)
            pairs += int(ok.sum())
            outs.append(_key(torch.cat([c[:, :1], o], 1)[ok], size).unique())
    return len(c), len(c) if stride == 1 else len(torch.cat(outs).unique()), pairs


def _geometry(case):
    return (case["k"], case["stride"], case["pad"]) if case["kind"] == "down" else (K, 1, 1)


def prepare(case, seed):
    config.allow_tf32 = case["dtype"] != "fp32_exact"
    dtype, res, batch, train = DTYPES[case["dtype"]], case["res"], case["batch"], case["train"]
    host = random.Random(seed)
    g = torch.Generator("cuda").manual_seed(seed)

    def normal(*shape, scale=1.0):
        return torch.randn(*shape, generator=g, device="cuda").mul_(scale).to(dtype)

    def leaf(t):
        return t.requires_grad_(train)

    # each object somewhere in its grid (even steps: the strided conv then has the same number of output rows everywhere)
    coords = _place(res, batch)
    free = res // 40
    moves = torch.tensor([[0] + [2 * host.randint(-free, free) for _ in range(3)] for _ in range(batch)], dtype=torch.int32, device="cuda")
    coords = coords + moves[coords[:, 0].long()]
    if case.get("shuffled"):
        coords = coords[torch.randperm(coords.shape[0], generator=g, device="cuda")].contiguous()
    n = coords.shape[0]

    if case["kind"] == "sample":
        per = case["points"] // batch
        rows = torch.bincount(coords[:, 0], minlength=batch).view(batch, 1)  # of each object: its points lie around its own voxels
        near = (torch.rand(batch, per, generator=g, device="cuda") * rows).long().clamp_(max=rows - 1) + rows.cumsum(0) - rows
        grid = coords[near, 1:] + 0.5 + torch.randn(batch, per, 3, generator=g, device="cuda") * 0.7
        s = dict(feats=leaf(normal(n, case["c"])), grid=grid, shape=torch.Size((batch, case["c"], res, res, res)))
        s["grad"] = normal(batch, per, case["c"]) if train else None
    else:
        k, stride, pad = _geometry(case)
        ci, co = (case["c"], case["c"]) if case["kind"] == "stack" else (case["ci"], case["co"])
        s = dict(feats=leaf(normal(n, ci)), shape=torch.Size((batch, ci, res, res, res)))
        s["layers"] = [(leaf(normal(co, k, k, k, ci, scale=(k ** 3 * ci) ** -0.5)), leaf(normal(co)) if case.get("bias", True) else None)
                       for _ in range(2 * case.get("blocks", 0) or 1)]
        s["grad"] = normal(_counts(res, batch, k, stride, pad)[1], co) if train else None
    s.update(case=case, coords=coords, cache=None)
    if case["kind"] == "conv" and not case["build"]:  # what an earlier layer of the network has left behind
        with torch.set_grad_enabled(train):
            s["cache"] = sparse_submanifold_conv3d(s["feats"], coords, s["shape"], *s["layers"][0])[1]
    return s


def _forward(s):
    case, feats, coords, shape = s["case"], s["feats"], s["coords"], s["shape"]
    if case["kind"] == "sample":
        return {"out": grid_sample_3d(feats, coords, shape, s["grid"], case["mode"])}
    weight, bias = s["layers"][0]
    if case["kind"] == "conv":
        out, cache = sparse_submanifold_conv3d(feats, coords, shape, weight, bias, s["cache"])
        return {"out": out, "map": cache["neighbor_map"].view(torch.int32)} if case["build"] else {"out": out}
    if case["kind"] == "down":
        k, stride, pad = _geometry(case)
        out, out_coords, _ = sparse_conv3d(feats, coords, shape, weight, bias, stride=(stride,) * 3, padding=(pad,) * 3)
        return {"out": out, "out_coords": out_coords}
    h, cache = feats, None
    for b in range(case["blocks"]):
        y, cache = sparse_submanifold_conv3d(h, coords, shape, *s["layers"][2 * b], cache)
        y, cache = sparse_submanifold_conv3d(torch.nn.functional.silu(y), coords, shape, *s["layers"][2 * b + 1], cache)
        h = h + y
    return {"out": h}


def run(s):
    if not s["case"]["train"]:
        with torch.no_grad():
            return _forward(s)
    got = _forward(s)
    leaves = [s["feats"]] + [t for layer in s.get("layers", ()) for t in layer if t is not None]
    got["grads"] = torch.autograd.grad(got["out"], leaves, s["grad"])
    got["out"] = got["out"].detach()
    return got


def work(case):
    size = DTYPES[case["dtype"]].itemsize
    train = case["train"]
    if case["kind"] == "sample":
        n = _counts(case["res"], case["batch"], K, 1, 1)[0]
        points = case["points"] // case["batch"] * case["batch"]
        corners = 8 if case["mode"] == "trilinear" else 1
        rows = min(n, points * corners)  # feature rows that can be touched
        return {"bytes": 16 * n + 12 * points + (rows + points) * case["c"] * size + (train and (points + n) * case["c"] * size),
                "flops": 2 * points * corners * case["c"] * (2 if train else 1)}
    k, stride, pad = _geometry(case)
    n, m, pairs = _counts(case["res"], case["batch"], k, stride, pad)
    ci, co = (case["c"], case["c"]) if case["kind"] == "stack" else (case["ci"], case["co"])
    convs = 2 * case.get("blocks", 0) or 1
    weights = k ** 3 * ci * co * size
    # activations and weights in and out of every conv: forward x, w -> y; backward dy, x, w -> dx, dw
    b = convs * (n * ci * size + m * co * size + weights + (train and 2 * n * ci * size + m * co * size + 2 * weights))
    b += 4 * k ** 3 * m  # the neighbour map, read where it is at hand and written where it is built
    if case["kind"] != "conv" or case["build"]:
        b += 16 * n
    if case["kind"] == "down":
        b += 16 * m + (train and 4 * k ** 3 * n)  # output coordinates, and the map of the backward direction
    return {"bytes": b, "flops": 2 * pairs * ci * co * convs * (3 if train else 1)}


def tolerance(case):
    # fp32 accumulation throughout; what differs is the rounding of the results (fp16 2^-11, bf16 2^-8), of the inputs
    # (TF32 2^-11) or the order of the sums and the split of the products (fp32-accurate)
    rel = {"fp16": 1e-3, "bf16": 5e-3, "fp32": 1e-3, "fp32_exact": 2e-5}[case["dtype"]]
    if case["kind"] == "sample" and case["dtype"] == "fp32":
        rel = 1e-5
    if case["kind"] == "stack":
        rel *= 2  # rounded again between the layers
    return {"rel": rel}
