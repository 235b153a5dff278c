"""The arc pass of the disk element takes 1 to 32 particles a warp, by how many have arcs: a particle's outputs are the same
bits alone, among a few and among many (148 SMs x 16 warps: one particle a warp up to 2368, 32 from 73 409 on)."""
import numpy as np
import pytest
import torch

from warpsphboundaries_b200.provider import FusedGroup, FusedWall
from warpsphboundaries_b200.scene import Body, DiskArrayRep, Scene
from warpsphboundaries_b200.shim import ParticleState

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["w4", "quintic"])
def test_same_bits_in_every_batch(kernel):
    rng = np.random.default_rng(17)
    C, R = rng.uniform(0, 1, (6, 2)), rng.uniform(0.02, 0.1, 6)
    C[:, 0] += np.arange(6)                                    # disks that do not overlap, one of them met by two arcs
    C[5] = C[4] + [R[4] + R[5] + 0.01, 0.0]
    n = 80_000
    j, t = rng.integers(0, 6, n), rng.uniform(0, 2 * np.pi, n)
    X = C[j] + (R[j] + rng.uniform(-0.04, 0.06, n))[:, None] * np.stack([np.cos(t), np.sin(t)], 1)
    sup = rng.uniform(0.03, 0.05, n)
    scene = Scene([Body(center=(0.3, 0.1), angle=0.4, reps=[DiskArrayRep(C, R)])], "cuda")
    c, s = np.cos(0.4), np.sin(0.4)
    W = torch.tensor(X @ np.array([[c, s], [-s, c]]) + [0.3, 0.1], device="cuda")
    S = torch.tensor(sup, device="cuda")

    def outputs(a, b):
        fw = FusedWall(scene, ParticleState(W[a:b].contiguous(), S[a:b].contiguous()), 0.05, (FusedGroup(kernel),))
        return {k: v[0] for k, v in fw.res[0].items()}

    whole = outputs(0, n)
    assert float((whole["lam"] > 0).double().mean()) > 0.6     # offsets of -0.04 .. 0.06, supports of 0.03 .. 0.05
    for m in (1, 31, 33, 2368, 2500, 40_000):
        part = outputs(100, 100 + m)
        for k in whole:
            assert torch.equal(part[k], whole[k][100:100 + m]), (m, k)
