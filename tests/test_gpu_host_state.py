"""State that the native host path shares between calls: the slots through which a build reports to the host."""
import pytest
import torch


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
