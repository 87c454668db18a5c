"""What the native host path keeps or must refuse: the slots through which a build reports to the host, the work
counters of the conv kernels, inputs that autograd treats specially."""
import pytest
import torch

from oracle import submconv_oracle as orc


pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def line(n):
    """n voxels in a row, and the grid around them."""
    z = torch.arange(n, dtype=torch.int32)
    return torch.stack([z * 0, z * 0, z * 0, z], 1).to(DEV).contiguous(), torch.Size((1, 8, 4, 4, n))


def test_host_slots_serve_every_kind_of_build_in_turn():
    """Builds of different kernel volumes report through the same slot one after the other.  Their counts fall while the
    number of uses of the slot rises, so a count left behind meets the number of a later use somewhere on the way."""
    from flexgemm_b200.ops.spconv import SubMConv3dFunction, sparse_conv3d
    feats = torch.randn(1500, 8, generator=torch.Generator().manual_seed(0)).half().to(DEV)
    w1, w8 = (torch.randn(8, *k, 8, generator=torch.Generator().manual_seed(1)).half().to(DEV).requires_grad_(True)
              for k in ((1, 1, 1), (1, 1, 8)))
    for n in range(1499, 8, -7):
        coords, shape = line(n)
        _, oc, cache = sparse_conv3d(feats[:n], coords, shape, w1)
        assert torch.equal(oc, coords) and cache["valid_signal_i"].shape[0] == n
        _, oc, cache = sparse_conv3d(feats[:n], coords, shape, w8, stride=(1, 1, 8))
        assert oc.shape[0] == n // 8 and cache["valid_signal_i"].shape[0] == n // 8 * 8
        cache = SubMConv3dFunction._compute_neighbor_cache(coords, shape, (1, 1, 5), (1, 1, 1), True)
        pairs = n + 2 * (n - 1) + 2 * (n - 2)
        assert cache["valid_signal_i"].shape[0] == pairs and cache["valid_signal_o"].shape[0] == pairs


@pytest.mark.parametrize("dtype", ["float16", "float32"])
def test_graph_replays_follow_their_inputs(dtype):
    """A captured pass gives on every replay what the same call gives outside a graph, also when the capturing stream has
    been used before, when several graphs are captured on it and when calls outside them come between."""
    from flexgemm_b200.kernels import cuda as K
    from flexgemm_b200.ops import spconv
    coords, feats, weight, bias, shape = (t.to(DEV) if torch.is_tensor(t) else t for t in orc.make_problem(16, 32, 96, dtype, seed=4))
    shape = torch.Size(shape)
    g = torch.Generator().manual_seed(9)
    gout = torch.randn(len(coords), 96, generator=g).to(feats.dtype).to(DEV)
    w = weight.detach().requires_grad_(True)
    x = feats.detach().clone().requires_grad_(True)
    _, cache = spconv.sparse_submanifold_conv3d(x, coords, shape, w, bias)

    def train():
        out, _ = spconv.sparse_submanifold_conv3d(x, coords, shape, w, bias, cache)
        return (out.detach(), *torch.autograd.grad(out, (x, w), gout))

    def infer():
        args = (x.detach(), coords, shape, w.detach(), bias)   # the first builds an inference cache, which waits for nothing
        return spconv.sparse_submanifold_conv3d(*args)[0], spconv.sparse_submanifold_conv3d(*args, cache)[0]

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            train(), infer()
    torch.cuda.current_stream().wait_stream(side)
    graphs = []
    for call in (train, infer, train):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            outs = call()
        graphs.append((graph, call, outs))
    for i in range(3):
        with torch.no_grad():
            x.copy_(torch.randn(x.shape, generator=g).to(x.dtype))
        for graph, call, outs in graphs:
            for o in outs:
                o.fill_(float("nan"))
            graph.replay()
            for got, want in zip(outs, call()):
                assert torch.equal(got, want)
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            train()
        torch.cuda.synchronize()
    K.check_status(DEV)


def test_work_counters_of_threads_on_one_stream():
    """Two threads run passes on the same stream, their backward passes beside the other's forward ones, through several
    refills of the counter pool and with more streams than it keeps pools for: every pass gives the same bits."""
    import threading

    from flexgemm_b200.kernels import cuda as K
    from flexgemm_b200.ops import spconv
    coords, feats, weight, bias, shape = (t.to(DEV) if torch.is_tensor(t) else t for t in orc.make_problem(12, 16, 32, "float16", seed=6))
    shape = torch.Size(shape)
    gout = torch.randn(len(coords), 32, generator=torch.Generator().manual_seed(3)).half().to(DEV)
    _, cache = spconv.sparse_submanifold_conv3d(feats, coords, shape, weight.detach().requires_grad_(True), bias)

    def once():
        x, w = feats.detach().requires_grad_(True), weight.detach().requires_grad_(True)
        out, _ = spconv.sparse_submanifold_conv3d(x, coords, shape, w, bias, cache)
        return (out.detach(), *torch.autograd.grad(out, (x, w), gout))
    want = once()
    torch.cuda.synchronize()
    wrong = []

    def work(seed):
        for i in range(400):
            if i % 6 == seed:
                with torch.cuda.stream(torch.cuda.ExternalStream(streams[(i + 31 * seed) % len(streams)].cuda_stream)):
                    once()
            got = once()
            if i % 8 == 0 and not all(torch.equal(a, b) for a, b in zip(got, want)):
                wrong.append((seed, i))
    streams = [torch.cuda.Stream(priority=p) for p in (0, -1) for _ in range(32)] + [torch.cuda.current_stream()]
    threads = [threading.Thread(target=work, args=(s,)) for s in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not wrong
    K.check_status(DEV)


@pytest.mark.parametrize("which", [0, 1, 2])
def test_forward_mode_is_refused(which):
    """There is no forward-mode derivative: a tangent on any input is an error, not an output without one."""
    import torch.autograd.forward_ad as fwad

    from flexgemm_b200.ops import grid_sample, spconv
    coords, *args, shape = (t.to(DEV) if torch.is_tensor(t) else t for t in orc.make_problem(8, 16, 16, "float16", seed=2))
    shape = torch.Size(shape)
    _, cache = spconv.sparse_submanifold_conv3d(args[0], coords, shape, args[1], args[2])
    query = torch.rand(1, 50, 3, device=DEV) * 8
    with fwad.dual_level():
        args[which] = fwad.make_dual(args[which], torch.ones_like(args[which]))
        f, w, b = args
        calls = [lambda: spconv.sparse_submanifold_conv3d(f, coords, shape, w, b), lambda: spconv.sparse_submanifold_conv3d(f, coords, shape, w, b, cache),
                 lambda: spconv.sparse_conv3d(f, coords, shape, w, b, stride=(2, 2, 2), padding=(1, 1, 1))]
        if which == 0:
            calls += [lambda: grid_sample.grid_sample_3d(f, coords, shape, query, "trilinear"),
                      lambda: grid_sample.grid_sample_3d(f, coords, shape, query, "nearest")]
        if which == 1:
            q = fwad.make_dual(query, torch.ones_like(query))
            calls.append(lambda: grid_sample.grid_sample_3d(args[0], coords, shape, q))
        for call in calls:
            with pytest.raises(NotImplementedError, match="jvp"):
                call()


@pytest.mark.parametrize("mode", ["trilinear", "nearest"])
def test_grid_sample_saves_its_map_as_autograd_does(mode):
    """The map of a sample is a saved tensor: freed by the backward pass (a second one is an error), kept by retain_graph,
    and seen by saved-tensor hooks.  (The order of the fp32 sums is not fixed: two passes may differ by one step of fp16.)"""
    from flexgemm_b200.ops import grid_sample
    coords, feats, _, _, shape = (t.to(DEV) if torch.is_tensor(t) else t for t in orc.make_problem(8, 16, 16, "float16", seed=2))
    feats.requires_grad_(True)
    query = torch.rand(1, 5000, 3, device=DEV) * 8
    (want,) = torch.autograd.grad(grid_sample.grid_sample_3d(feats, coords, torch.Size(shape), query, mode).sum(), feats)
    out = grid_sample.grid_sample_3d(feats, coords, torch.Size(shape), query, mode).sum()
    for retain in (True, False):
        (got,) = torch.autograd.grad(out, feats, retain_graph=retain)
        assert torch.allclose(got, want, rtol=2e-3, atol=2e-3)
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(out, feats)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.numel()) or t.cpu(), lambda t: t.to(DEV)):
        out = grid_sample.grid_sample_3d(feats, coords, torch.Size(shape), query, mode)
    assert packed == ([40000, 40000] if mode == "trilinear" else [5000])
    (got,) = torch.autograd.grad(out.sum(), feats)
    assert torch.allclose(got, want, rtol=2e-3, atol=2e-3)
    held = torch.cuda.memory_allocated()
    out = grid_sample.grid_sample_3d(feats, coords, torch.Size(shape), query, mode)
    (got,) = torch.autograd.grad(out.sum(), feats)
    assert torch.cuda.memory_allocated() - held <= 2 * out.numel() + 4 * got.numel() + 4096   # the output and the gradient


@pytest.mark.parametrize("feats_grad", [False, True])
def test_grid_sample_with_query_points_that_require_grad(feats_grad):
    """There is no gradient with respect to the points, yet the output takes part in the graph."""
    from flexgemm_b200.ops import grid_sample
    coords, feats, _, _, shape = (t.to(DEV) if torch.is_tensor(t) else t for t in orc.make_problem(8, 16, 16, "float32", seed=2))
    feats.requires_grad_(feats_grad)
    query = (torch.rand(1, 50, 3, device=DEV) * 8).requires_grad_(True)
    out = grid_sample.grid_sample_3d(feats, coords, torch.Size(shape), query)
    assert out.requires_grad
    out.sum().backward()
    assert query.grad is None and (feats.grad is not None) == feats_grad


@pytest.mark.parametrize("op", ["submanifold", "strided"])
def test_backward_takes_the_fp32_setting_of_its_own_time(op):
    """TF32 or accurate fp32 is decided when a pass runs: a backward pass after the switch is the other pass's, bit for
    bit, and not this one's."""
    from flexgemm_b200.kernels import config
    from flexgemm_b200.kernels.triton.spconv import config as forwarded
    from flexgemm_b200.ops import spconv
    coords, feats, weight, bias, shape = (t.to(DEV) if torch.is_tensor(t) else t for t in orc.make_problem(8, 32, 32, "float32", seed=2))
    f, w = feats.requires_grad_(True), weight.requires_grad_(True)
    assert config.allow_tf32

    def grads(at_forward, at_backward):
        try:
            config.allow_tf32 = at_forward
            if op == "submanifold":
                out = spconv.sparse_submanifold_conv3d(f, coords, torch.Size(shape), w, bias)[0]
            else:
                out = spconv.sparse_conv3d(f, coords, torch.Size(shape), w, bias, stride=(2, 2, 2), padding=(1, 1, 1))[0]
            forwarded.allow_tf32 = at_backward
            return torch.autograd.grad(out, (f, w), torch.randn(out.shape, generator=torch.Generator().manual_seed(1)).to(DEV))
        finally:
            config.allow_tf32 = True
    tf32, exact = grads(True, True), grads(False, False)
    for got, want, other in zip(grads(True, False) + grads(False, True), exact + tf32, tf32 + exact):
        assert torch.equal(got, want) and not torch.equal(got, other)


def test_grids_that_no_key_can_hold_are_refused():
    """2^64 cells and more: an error from every entry point, and 2^63 cells go through."""
    from flexgemm_b200.ops import grid_sample, spconv
    coords, feats, weight, bias, _ = (t.to(DEV) if torch.is_tensor(t) else t for t in orc.make_problem(8, 16, 16, "float16", seed=2))
    query = torch.rand(1, 50, 3, device=DEV) * 8
    calls = [lambda s: spconv.sparse_submanifold_conv3d(feats, coords, s, weight, bias)[0], lambda s: grid_sample.grid_sample_3d(feats, coords, s, query),
             lambda s: spconv.sparse_conv3d(feats, coords, s, weight, bias, stride=(2 ** 16,) * 3, padding=(1, 1, 1))[0]]
    small = torch.Size((1, 16, 2 ** 21, 2 ** 21, 2 ** 21))
    for extents in ((2 ** 22, 2 ** 21, 2 ** 21), (2 ** 31 - 1,) * 3):
        for call in calls:
            with pytest.raises(ValueError, match="too large"):
                call(torch.Size((1, 16, *extents)))
    for call in calls:
        assert torch.isfinite(call(small)).all()
    assert torch.equal(calls[0](small), calls[0](torch.Size((1, 16, 8, 8, 8))))


def test_calls_that_fail_give_their_slot_back():
    """Builds that the library refuses after a slot was taken (coordinates that are not 16-byte aligned)."""
    from flexgemm_b200 import _native
    from flexgemm_b200.ops import spconv
    coords, feats, weight, bias, shape = (t.to(DEV) if torch.is_tensor(t) else t for t in orc.make_problem(8, 16, 16, "float16", seed=2))
    shape = torch.Size(shape)
    weight.requires_grad_(True)
    want = spconv.sparse_submanifold_conv3d(feats, coords, shape, weight, bias)[0]
    spconv.sparse_conv3d(feats, coords, shape, weight, bias, stride=(2, 2, 2), padding=(1, 1, 1))
    off = torch.empty(coords.numel() + 1, dtype=torch.int32, device=DEV)[1:].view(-1, 4)
    off.copy_(coords)
    made, free = _native.ext().host_slots()
    assert made == free and made > 0
    for _ in range(made + 1):
        with pytest.raises(ValueError, match="align"):
            spconv.sparse_submanifold_conv3d(feats, off, shape, weight, bias)
        with pytest.raises(ValueError, match="align"):
            spconv.sparse_conv3d(feats, off, shape, weight, bias, stride=(2, 2, 2), padding=(1, 1, 1))
    assert _native.ext().host_slots() == (made, free)
    assert torch.equal(spconv.sparse_submanifold_conv3d(feats, coords, shape, weight, bias)[0], want)


def test_strided_rows_of_a_batch_beyond_the_shape():
    """The hash path takes every batch index, so the bit grid, which has no place for one beyond the shape's, leaves the
    call to it: no output row is lost."""
    from flexgemm_b200.ops import spconv
    coords, feats, weight, bias, shape = (t.to(DEV) if torch.is_tensor(t) else t for t in orc.make_problem(9, 16, 16, "float32", seed=2, batch=3))
    geom = dict(stride=(2, 2, 2), padding=(1, 1, 1))
    outs = []
    for batches in (3, 2):
        w = weight.detach().requires_grad_(True)
        out, oc, _ = spconv.sparse_conv3d(feats, coords, torch.Size((batches, *shape[1:])), w, bias, **geom)
        (gw,) = torch.autograd.grad(out.sum(), w)
        only = spconv.SparseConv3dFunction._get_output_coords(coords, torch.Size((batches, *shape[1:])), (3, 3, 3), (2, 2, 2), (1, 1, 1), (1, 1, 1))
        key, also = (((c[:, 0].long() * 64 + c[:, 1]) * 64 + c[:, 2]) * 64 + c[:, 3] for c in (oc, only))
        assert torch.equal(key.sort().values, also.sort().values)   # the order of such rows is not fixed
        outs.append((key.sort().values, out.detach()[key.argsort()], gw))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    # the pairs of an offset are summed in row order, which differs: fp32 sums of TF32 products
    assert (outs[0][2] - outs[1][2]).abs().max() <= 1e-5 * outs[0][2].abs().max() * len(key) ** 0.5


def test_launch_count_follows_the_kernels_that_run():
    """The count is taken where kernels are launched, so it follows the path a call takes."""
    from flexgemm_b200.kernels import cuda as K
    from flexgemm_b200.ops import grid_sample, spconv
    coords, feats, weight, bias, shape = (t.to(DEV) if torch.is_tensor(t) else t for t in orc.make_problem(8, 64, 64, "float16", seed=2))
    shape = torch.Size(shape)
    f, w = feats.requires_grad_(True), weight.requires_grad_(True)

    def launches(call):
        before = K.launch_count
        out = call()
        return K.launch_count - before, out
    prev = K.set_conv_splitk(1)
    try:
        geom = (coords, shape, (3, 3, 3), (1, 1, 1))
        assert launches(lambda: spconv.SubMConv3dFunction._compute_neighbor_cache(*geom, False))[0] == 2   # map, plan
        count, cache = launches(lambda: spconv.SubMConv3dFunction._compute_neighbor_cache(*geom, True))
        assert count == 3                                                                                  # and the pair lists
        count, (out, _) = launches(lambda: spconv.sparse_submanifold_conv3d(f, coords, shape, w, bias, cache))
        assert count == 1
        assert launches(lambda: torch.autograd.grad(out, f, torch.ones_like(out), retain_graph=True))[0] == 1   # weight read as stored
        # marking, counting, coordinates, maps, codes, plan, pair lists, convolution
        assert launches(lambda: spconv.sparse_conv3d(f, coords, shape, w, bias, stride=(2, 2, 2), padding=(1, 1, 1)))[0] == 8
        count, out = launches(lambda: grid_sample.grid_sample_3d(f, coords, shape, torch.rand(1, 100, 3, device=DEV) * 8))
        assert count == 2
        assert launches(lambda: torch.autograd.grad(out, f, torch.ones_like(out)))[0] == 4
    finally:
        K.set_conv_splitk(prev)
