"""Closed surfaces, more queries than one slice of the workspace: the same bits as calls on the parts, with and without the
inside flags, and a workspace that no longer grows."""
import numpy as np
import pytest
import torch

from warpsphboundaries_b200 import _lib
from warpsphboundaries_b200 import workloads as W
from warpsphboundaries_b200.mesh3d import ClosedMesh

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")
SLICE = 1 << 22


def test_workspace_is_bounded():
    mesh = ClosedMesh(*W.icosphere(2, 0.6), 0.1, DEV)
    size = lambda n: int(_lib.lib.wsb_mesh_workspace_size(mesh.handle, n))
    assert size(1000) < size(SLICE) == size(SLICE + 1) == size(1 << 28) <= 12 << 28


@pytest.mark.parametrize("over", [1, 70_001])
def test_slices_give_the_bits_of_their_parts(over):
    n = SLICE + over
    mesh = ClosedMesh(*W.icosphere(2, 0.6, 0.05, seed=2), 0.1, DEV)
    g = torch.Generator(device=DEV)
    g.manual_seed(8)
    pos = 1.6 * torch.rand((n, 3), dtype=torch.float64, device=DEV, generator=g) - 0.8
    sup = 0.05 + 0.05 * torch.rand(n, dtype=torch.float64, device=DEV, generator=g)
    sup[7::100_003] = 0.2                                         # beyond the grid's supports: NaN rows
    inside = torch.empty(n, dtype=torch.int32, device=DEV)
    whole = mesh.channels(pos, sup, "w4", inside=inside)
    bits = lambda t: t.view(torch.int64)
    for a, b in ((0, SLICE), (SLICE, n), (SLICE - 5, SLICE + over)):
        flags = torch.empty(b - a, dtype=torch.int32, device=DEV)
        assert torch.equal(bits(mesh.channels(pos[a:b], sup[a:b], "w4", inside=flags)), bits(whole[a:b]))
        assert torch.equal(flags, inside[a:b])
    assert torch.equal(bits(mesh.channels(pos, sup, "w4")), bits(whole))
    assert int((inside < 0).sum()) == len(range(7, n, 100_003)) and bool(torch.isnan(whole[7]).all())
