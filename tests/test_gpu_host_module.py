"""The native host path against the library's single-purpose calls: cache build (map, order, masks, schedule, pair lists)
at the edges of its tiles, the bias gradient computed along with the weight gradient, and padded channel counts."""
import numpy as np
import pytest
import torch

from oracle import submconv_oracle as orc

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def u32(t):
    return t.cpu().view(torch.int32).numpy().view(np.uint32)


@pytest.mark.parametrize("n,ksize,shuffle,volume", [(1, (3, 3, 3), False, 64), (127, (3, 3, 3), False, 64), (128, (3, 3, 3), True, 64),
                                                    (257, (3, 1, 3), False, 64), (1025, (3, 3, 3), True, 64), (4097, (1, 1, 1), False, 64),
                                                    (8192, (3, 3, 3), True, 64), (8193, (3, 3, 3), False, 64), (2049, (3, 1, 1), True, 2048), (33000, (3, 3, 3), False, 64), (33000, (3, 3, 3), True, 2048),
                                                    (131071, (3, 3, 3), True, 64), (131072, (3, 3, 3), True, 64), (131073, (3, 1, 3), False, 64), (140001, (3, 3, 3), True, 2048),
                                                    (3000, (1, 1, 31), False, 64), (1, (1, 1, 1), False, 64)])
def test_cache_build_matches_single_calls(n, ksize, shuffle, volume):
    from flexgemm_b200.kernels import cuda as K
    from flexgemm_b200.ops import utils
    from flexgemm_b200.ops.spconv import SubMConv3dFunction
    g = torch.Generator().manual_seed(n)
    flat = torch.randperm(64 ** 3, generator=g)[:n].sort().values
    coords = torch.stack([flat * 0, flat // 4096, flat // 64 % 64, flat % 64], 1).int()
    if shuffle:
        coords = coords[torch.randperm(n, generator=g)]
    coords = coords.to(DEV).contiguous()
    shape = torch.Size((1, 8, volume, volume, volume))
    V = ksize[0] * ksize[1] * ksize[2]
    got = SubMConv3dFunction._compute_neighbor_cache(coords, shape, ksize, (1, 1, 1), True)
    table, bits = utils.init_table(shape, max(2 * n, 1), DEV)
    want = K.subm_build_neighbor_map(coords, shape, ksize, (1, 1, 1), table, bits, max(2 * n, 1))
    seg = u32(want["valid_signal_seg"])
    order = K.sorted_idx_from_binary(want["binary_code"], V)
    vs_i, vs_o = K.valid_signal(want["neighbor_map"], want["gray_code"], want["block_offsets"], want["valid_signal_seg"], int(seg[V]))
    masks = K.tile_masks(want["gray_code"], order, 128)
    for name, ref in (("neighbor_map", want["neighbor_map"]), ("valid_signal_seg", want["valid_signal_seg"]), ("valid_signal_i", vs_i),
                      ("valid_signal_o", vs_o), ("pair_block_offsets", want["block_offsets"]), ("tile_masks_128", masks)):
        assert np.array_equal(u32(got[name]), u32(ref)), name
    assert torch.equal(got["gray_code"], want["gray_code"]) and torch.equal(got["sorted_idx"], order)
    # a schedule is any order of descending cost
    m = u32(masks)
    m = np.concatenate([m, np.zeros(len(m) % 2, np.uint32)]).reshape(-1, 2)
    cost = np.array([bin(int(a)).count("1") + bin(int(b)).count("1") for a, b in m])
    blocks = u32(got["block_order_128"])
    assert np.array_equal(np.sort(blocks), np.arange(len(cost))) and np.all(np.diff(cost[blocks]) <= 0)
    K.check_status(DEV)


@pytest.mark.parametrize("res,ci,co,dtype", [(8, 8, 8, "float16"), (16, 6, 20, "bfloat16"), (16, 32, 136, "float16"), (8, 3, 1032, "float32"),
                                             (24, 64, 2056, "bfloat16")])
def test_gradients_with_bias_and_padding(res, ci, co, dtype):
    """The bias sums are fp32 over at most a few thousand values and rounded once: within half a unit in the last place
    of the type plus n * 2^-24 of the absolute sum; everything else within the library's 1e-2 of the oracle's maximum."""
    from flexgemm_b200.ops import spconv
    coords, feats, weight, bias, shape = orc.make_problem(res, ci, co, dtype, seed=res + co)
    gout = torch.randn(coords.shape[0], co, generator=torch.Generator().manual_seed(1)).to(feats.dtype)
    f, w, b = (t.to(DEV).requires_grad_(True) for t in (feats, weight, bias))
    out, cache = spconv.sparse_submanifold_conv3d(f, coords.to(DEV), torch.Size(shape), w, b)
    gf, gw, gb = torch.autograd.grad(out, (f, w, b), gout.to(DEV))
    nbr = orc.neighbor_map(coords.numpy(), shape)
    rf, rw, rb = orc.conv_backward(gout.double(), feats.double(), nbr, weight.double())
    ro = orc.conv_forward(feats.double(), nbr, weight.double(), bias.double())
    for got, want in ((out, ro), (gf, rf), (gw, rw)):
        assert (got.detach().cpu().double() - want).abs().max() <= 1e-2 * want.abs().max()
    ulp = {"float16": 2.0 ** -11, "bfloat16": 2.0 ** -8, "float32": 2.0 ** -24}[dtype]
    bound = rb.abs() * ulp + gout.double().abs().sum(0) * 2.0 ** -24 * gout.shape[0] + 1e-7
    assert torch.all((gb.cpu().double() - rb).abs() <= bound)
    # the same through the Python autograd function
    out2, _ = spconv.SubMConv3dFunction.apply(f, coords.to(DEV), torch.Size(shape), cache, w, b)
    for x, y in zip((out2, *torch.autograd.grad(out2, (f, w, b), gout.to(DEV))), (out, gf, gw, gb)):
        assert torch.equal(x, y)


def test_inference_cache_has_no_pair_lists():
    from flexgemm_b200.ops import spconv
    coords, feats, weight, bias, shape = orc.make_problem(8, 16, 16, "float16", seed=3)
    _, cache = spconv.sparse_submanifold_conv3d(feats.to(DEV), coords.to(DEV), torch.Size(shape), weight.to(DEV), bias.to(DEV))
    w = weight.to(DEV).requires_grad_(True)
    out, _ = spconv.sparse_submanifold_conv3d(feats.to(DEV), coords.to(DEV), torch.Size(shape), w, None, cache)
    with pytest.raises(AttributeError, match="valid_signal_i"):
        out.sum().backward()


@pytest.mark.parametrize("C,dtype,mode,points", [(4, "float16", "trilinear", 1), (12, "bfloat16", "trilinear", 37), (64, "float16", "nearest", 1000),
                                                 (136, "float32", "trilinear", 333), (256, "bfloat16", "trilinear", 515), (264, "float16", "nearest", 130),
                                                 (520, "float16", "trilinear", 77), (72, "float32", "trilinear", 60000), (8, "float16", "nearest", 40000)])
@pytest.mark.parametrize("volume", [16, 2048])
def test_grid_sample_matches_separate_kernels(C, dtype, mode, points, volume):
    """Forward: the same bits as the map kernel followed by the gather (same weights, fp32 sums over the corners in the
    same order; only the fused multiply-adds may be contracted differently: one rounding step of the type).  Gradient:
    fp32 sums of the same terms in another order, up to `terms` of them, then one rounding."""
    from flexgemm_b200.kernels import cuda as K
    from flexgemm_b200.ops import grid_sample, utils
    T = getattr(torch, dtype)
    coords = torch.from_numpy(orc.make_problem(16, 8, 8, "float16", seed=5, batch=2)[0].numpy()).to(DEV)
    shape = torch.Size((2, C, volume, volume, volume))
    g = torch.Generator().manual_seed(C)
    feats = torch.randn(coords.shape[0], C, generator=g).to(T).to(DEV).requires_grad_(True)
    query = (torch.rand(2, points, 3, generator=g) * 18 - 1).to(DEV)
    gout = torch.randn(2, points, C, generator=g).to(T).to(DEV)
    out = grid_sample.grid_sample_3d(feats, coords, shape, query, mode)
    (gf,) = torch.autograd.grad(out, feats, gout)
    slots = 2 * coords.shape[0]
    table, bits = utils.init_table(shape, slots, DEV)
    K.table_insert_3d_idx_as_val(table, bits, slots, coords, volume, volume, volume)
    nb = K.grid_sample_neighbor_map(table, bits, slots, query, volume, volume, volume, mode == "trilinear")
    idx, w = (nb[0].view(-1, 8), nb[1].view(-1, 8)) if mode == "trilinear" else (nb.view(-1, 1), None)
    want = K.indice_weighted_sum_fwd(feats.detach(), idx, w).view(out.shape)
    ulp = {"float16": 2.0 ** -10, "bfloat16": 2.0 ** -7, "float32": 2.0 ** -22}[dtype]
    assert torch.all((out.detach().double() - want.double()).abs() <= want.double().abs() * ulp + 1e-6)
    g32 = K.indice_weighted_sum_bwd(gout.view(-1, C), idx, w, coords.shape[0]).double()
    mag = K.indice_weighted_sum_bwd(gout.view(-1, C).abs(), idx, w, coords.shape[0]).double()
    terms = 8.0 * points / 100
    assert torch.all((gf.double() - g32).abs() <= g32.abs() * ulp + mag * 2.0 ** -24 * (2 + terms) + 1e-7)


@pytest.mark.parametrize("ksize,stride,pad,dil", [((2, 2, 2), (2, 2, 2), (0, 0, 0), (1, 1, 1)), ((3, 3, 3), (2, 2, 2), (1, 1, 1), (1, 1, 1)),
                                                  ((3, 1, 2), (1, 3, 2), (2, 0, 1), (2, 1, 1)), ((1, 1, 1), (1, 1, 1), (0, 0, 0), (1, 1, 1)),
                                                  ((1, 1, 32), (1, 1, 4), (0, 0, 15), (1, 1, 1))])
@pytest.mark.parametrize("n,shuffle", [(1, False), (255, True), (3000, False), (8192, True), (40000, True)])
def test_strided_build_matches_hash_path(ksize, stride, pad, dil, n, shuffle):
    """Output coordinates and maps made on the bit grid against the hash set, sort and table of the generic calls."""
    from flexgemm_b200 import _native
    from flexgemm_b200.kernels import cuda as K
    from flexgemm_b200.ops import utils
    from flexgemm_b200.ops.spconv import SparseConv3dFunction, SparseConv3dNeighborCache, sparse_conv3d
    g = torch.Generator().manual_seed(n)
    W, H, D = 40, 33, 70
    flat = torch.randperm(2 * W * H * D, generator=g)[:n].sort().values
    coords = torch.stack([flat // (W * H * D), flat // (H * D) % W, flat // D % H, flat % D], 1).int()
    if shuffle:
        coords = coords[torch.randperm(n, generator=g)]
    coords = coords.to(DEV).contiguous()
    shape = torch.Size((2, 8, W, H, D))
    geom = (shape, ksize, stride, pad, dil)
    want_oc = K.sparse_out_coords(coords, *geom, 1.1, 0)
    assert torch.equal(SparseConv3dFunction._get_output_coords(coords, *geom), want_oc)
    on_bits = _native.ext().strided_coords(coords, *geom)   # None where the call is left to the hash path
    assert on_bits is not None and torch.equal(on_bits, want_oc)
    feats = torch.randn(n, 8, generator=g).half().to(DEV).requires_grad_(True)
    weight = torch.randn(8, *ksize, 8, generator=g).half().to(DEV)
    native = _native.ext().strided_conv(SparseConv3dNeighborCache, feats, coords, shape, weight, None, stride, pad, dil, True)
    if want_oc.shape[0] == 0:
        assert native is None and sparse_conv3d(feats, coords, shape, weight, None, stride=stride, padding=pad, dilation=dil)[0].shape == (0, 8)
        return
    out, oc, cache = native
    assert torch.equal(oc, want_oc) and out.shape == (oc.shape[0], 8)
    assert torch.equal(sparse_conv3d(feats, coords, shape, weight, None, stride=stride, padding=pad, dilation=dil)[0], out)
    V = ksize[0] * ksize[1] * ksize[2]
    table, bits = utils.init_table(shape, max(2 * n, 1), DEV)
    want = K.sparse_build_neighbor_map(coords, oc, *geom, table, bits, max(2 * n, 1), True)
    seg = u32(want["valid_signal_seg"])
    vs_i, vs_o = K.valid_signal(want["neighbor_map"], want["gray_code"], want["block_offsets"], want["valid_signal_seg"], int(seg[V]))
    gray_bwd, binary_bwd = K.gray_code_from_map(want["neighbor_map_bwd"])
    order, order_bwd = K.sorted_idx_from_binary(want["binary_code"], V), K.sorted_idx_from_binary(binary_bwd, V)
    for name, ref in (("neighbor_map", want["neighbor_map"]), ("neighbor_map_bwd", want["neighbor_map_bwd"]), ("valid_signal_i", vs_i),
                      ("valid_signal_o", vs_o), ("valid_signal_seg", want["valid_signal_seg"]), ("pair_block_offsets", want["block_offsets"]),
                      ("tile_masks_128", K.tile_masks(want["gray_code"], order, 128)), ("tile_masks_bwd_128", K.tile_masks(gray_bwd, order_bwd, 128))):
        assert np.array_equal(u32(cache[name]), u32(ref)), name
    for name, ref in (("gray_code", want["gray_code"]), ("gray_code_bwd", gray_bwd), ("sorted_idx", order), ("sorted_idx_bwd", order_bwd)):
        assert torch.equal(cache[name], ref), name
    K.check_status(DEV)


@pytest.mark.parametrize("n,co,dtype", [(148 * 256 + 1, 32, "float16"), (150 * 256, 64, "bfloat16"), (163 * 128 + 37, 264, "float32"), (222 * 256 - 5, 16, "float16")])
def test_halved_items_at_the_end_of_a_launch(n, co, dtype):
    """Launches whose last work items go out as halves: bit for bit the rows of the same convolution with the number of
    SMs capped so that no item is halved."""
    from flexgemm_b200.kernels import cuda as K
    from flexgemm_b200.ops.spconv import sparse_submanifold_conv3d
    T = getattr(torch, dtype)
    g = torch.Generator().manual_seed(n)
    flat = torch.randperm(96 ** 3, generator=g)[:n].sort().values
    coords = torch.stack([flat * 0, flat // 96 ** 2, flat // 96 % 96, flat % 96], 1).int().to(DEV).contiguous()
    shape = torch.Size((1, 32, 96, 96, 96))
    feats = torch.randn(n, 32, generator=g).to(T).to(DEV).requires_grad_(True)
    weight = (torch.randn(co, 3, 3, 3, 32, generator=g) / 12).to(T).to(DEV)
    gout = torch.randn(n, co, generator=g).to(T).to(DEV)
    out, cache = sparse_submanifold_conv3d(feats, coords, shape, weight)
    (gf,) = torch.autograd.grad(out, feats, gout)
    prev = K.set_conv_cta_limit(7)          # more than six waves: nothing is halved
    try:
        out1, _ = sparse_submanifold_conv3d(feats, coords, shape, weight, None, cache)
        (gf1,) = torch.autograd.grad(out1, feats, gout)
    finally:
        K.set_conv_cta_limit(prev)
    assert torch.equal(out, out1) and torch.equal(gf, gf1)
    K.check_status(DEV)


@pytest.mark.parametrize("res,ci,co,dtype,tf32", [(8, 40, 40, "float16", True), (8, 1024, 264, "bfloat16", True), (16, 512, 1024, "float16", True),
                                                  (8, 136, 300, "float32", True), (8, 260, 132, "float32", False), (2, 16, 16, "float16", True)])
def test_weight_gradient_without_slabs(res, ci, co, dtype, tf32):
    """Every offset as one unit that writes its result directly, against slabs and their ordered sum: the same products,
    summed in fp32 in another grouping.  The kernels launched show which way a call took."""
    from flexgemm_b200.kernels import config
    from flexgemm_b200.kernels import cuda as K
    from flexgemm_b200.ops import spconv
    coords, feats, weight, bias, shape = orc.make_problem(res, ci, co, dtype, seed=res + co)
    config.allow_tf32 = tf32
    got, launches = {}, {}
    try:
        f, w, b = (t.to(DEV).requires_grad_(True) for t in (feats, weight, bias))
        gout = torch.randn(coords.shape[0], co, generator=torch.Generator().manual_seed(2)).to(f.dtype).to(DEV)
        for mode in (1, 2, 0):
            K.set_wgrad_direct(mode)
            out, cache = spconv.sparse_submanifold_conv3d(f, coords.to(DEV), torch.Size(shape), w, b)
            before = K.launch_count
            got[mode] = torch.autograd.grad(out, (w, b), gout)
            launches[mode] = K.launch_count - before
        _, gw32 = K.conv_wgrad(gout, f.detach(), cache["valid_signal_i"], cache["valid_signal_o"], cache["valid_signal_seg"], want_f32=True)
        gb32 = K.bias_grad(gout, want_f32=True)[1]
    finally:
        K.set_wgrad_direct(0)
        config.allow_tf32 = True
    passes = 1 if tf32 or dtype != "float32" else 3
    assert launches[2] == launches[1] + passes and launches[0] in (launches[1], launches[2])
    ulp = {"float16": 2.0 ** -11, "bfloat16": 2.0 ** -8, "float32": 2.0 ** -24}[dtype]
    for gw, gb in got.values():
        for x, want, terms in ((gw.view(co, 27, ci), gw32, 27 + len(coords)), (gb, gb32, len(coords))):
            err = (x.double() - want.double()).abs()
            assert torch.all(err <= want.double().abs() * ulp + want.double().abs().max() * terms * 2.0 ** -24 + 1e-7)
    K.check_status(DEV)


@pytest.mark.parametrize("dtype", ["float16", "float32"])
@pytest.mark.parametrize("ci,co", [(8, 8), (16, 40), (40, 72), (72, 136), (96, 96), (136, 200), (200, 320), (264, 312), (520, 16)])
def test_channel_tiles_of_any_width(ci, co, dtype):
    """Column tiles, accumulator blocks and chunks at widths off the powers of two, forward and backward, against the
    oracle; RES=20 has enough rows for two blocks and takes every slice of the reduction."""
    from flexgemm_b200.kernels import cuda as K
    from flexgemm_b200.ops import spconv
    coords, feats, weight, bias, shape = orc.make_problem(20, ci, co, dtype, seed=ci + co)
    gout = torch.randn(coords.shape[0], co, generator=torch.Generator().manual_seed(2)).to(feats.dtype)
    nbr = orc.neighbor_map(coords.numpy(), shape)
    want = (orc.conv_forward(feats.double(), nbr, weight.double(), bias.double()),
            *orc.conv_backward(gout.double(), feats.double(), nbr, weight.double()))
    for splits in (0, 1):
        prev = K.set_conv_splitk(splits)
        try:
            f, w, b = (t.to(DEV).requires_grad_(True) for t in (feats, weight, bias))
            out, cache = spconv.sparse_submanifold_conv3d(f, coords.to(DEV), torch.Size(shape), w, b)
            got = (out, *torch.autograd.grad(out, (f, w, b), gout.to(DEV)))
            # the weight gradient through slabs as well
            gw, _ = K.conv_wgrad(gout.to(DEV), f.detach(), cache["valid_signal_i"], cache["valid_signal_o"], cache["valid_signal_seg"], splitk=3,
                                 want_f32=True)
        finally:
            K.set_conv_splitk(prev)
        for x, y in zip((*got, gw.view(want[2].shape)), (*want, want[2])):
            assert (x.detach().cpu().double() - y).abs().max() <= 1e-2 * y.abs().max()
    K.check_status(DEV)
