"""Rows of 32 pairs and more in passes of two, three and four kernels: their eight lanes' sums are added up channel by
channel (24, 36 and 48 of them, eight at a time), so every channel of every kernel is compared with the kernel's own pass.
The same pairs and the same closed forms in both; the tolerance of 1e-12 in units of the support allows another order of
some hundred additions and the packs' shared special functions (1e-13 in the group tests, for rows of a few pairs)."""
import numpy as np
import pytest
import torch

from tests.helpers import DEV, make_scene
from warpsphboundaries_b200.provider import FusedGroup, FusedWall
from warpsphboundaries_b200.shim import ParticleState

pytestmark = pytest.mark.gpu
H = 0.05


@pytest.mark.parametrize("kernels", [("w4", "cone"), ("w2", "cone", "lw2"), ("w2", "w4", "w6"), ("cubic", "w2", "w4", "w6")])
@pytest.mark.parametrize("n", [700, 150_000])
def test_pack_equals_its_kernels(kernels, n):
    t = np.concatenate([np.linspace(0, 3.0, 1600, endpoint=False), np.linspace(3.0, 2 * np.pi, 200, endpoint=False)])
    ring = np.stack([0.5 * np.cos(t), 0.5 * np.sin(t)], 1)
    rng = np.random.default_rng(n)
    a, r = rng.uniform(0, 2 * np.pi, n), 0.5 + H * rng.uniform(-1.1, 1.1, n)
    scene, _, _ = make_scene([ring], center=(0.1, -0.2), angle=0.4)
    c, s = np.cos(0.4), np.sin(0.4)
    X = np.stack([r * np.cos(a), r * np.sin(a)], 1) @ np.array([[c, s], [-s, c]]) + np.array([0.1, -0.2])
    ps = ParticleState(torch.tensor(X, device=DEV), torch.full((n,), H, dtype=torch.float64, device=DEV))
    pack = FusedWall(scene, ps, H, tuple(FusedGroup(k) for k in kernels)).res
    unit = {"lam": 1.0, "G": H, "Cov": 1.0, "m1": 1 / H, "m2": 1 / H ** 2}
    for g, k in enumerate(kernels):
        alone = FusedWall(scene, ps, H, (FusedGroup(k),)).res[0]
        for q, u in unit.items():
            assert float(((pack[g][q] - alone[q]) * u).abs().max()) <= 1e-12, (k, q)
