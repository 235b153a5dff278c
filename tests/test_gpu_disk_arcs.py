"""The arc pass of the disk element: particles listed by their number of arcs (none, one, several), each arc cut into
items of 12 nodes over a warp's lanes.

Particles that meet no, one and up to a dozen circles, or lie inside a covering disk as well: alone and among others the
same bits, and against the oracle's adaptive quadrature within 1e-10 in units of the support (its own accuracy, as for the
bundle tests).  One kernel without knots, one with one, one with two."""
import numpy as np
import pytest
import torch

from oracle import disk as Dk
from oracle import edge2d as O
from warpsphboundaries_b200.provider import FusedGroup, FusedWall
from warpsphboundaries_b200.scene import Body, DiskArrayRep, Scene
from warpsphboundaries_b200.shim import ParticleState

pytestmark = pytest.mark.gpu
DEV, H = "cuda", 0.1
NAMES = ("lam", "G", "Cov", "m1", "m2")


def _scene():
    """a 5 x 5 lattice of small disks (radius 0.2 H, spacing 0.45 H), one large disk, one far larger than the support."""
    g = np.stack(np.meshgrid(np.arange(5), np.arange(5)), -1).reshape(-1, 2) * 0.45 * H
    C = np.concatenate([g, [[0.9, 0.1], [-0.8, 0.0]]])
    R = np.concatenate([np.full(25, 0.2 * H), [0.15, 0.5]])
    return C, R


def _wall(X, kernel):
    C, R = _scene()
    scene = Scene([Body(reps=[DiskArrayRep(C, R)])], DEV)
    ps = ParticleState(torch.tensor(X, dtype=torch.float64, device=DEV), torch.full((len(X),), H, dtype=torch.float64, device=DEV))
    fw = FusedWall(scene, ps, H, (FusedGroup(kernel),))
    return {k: fw.res[0][k][0].cpu().numpy() for k in NAMES}


@pytest.mark.parametrize("kernel", ["w4", "cubic", "quintic"])
def test_every_number_of_arcs(kernel):
    C, R = _scene()
    rng = np.random.default_rng(17)
    X = np.concatenate([rng.uniform(-0.1, 0.28, (90, 2)), rng.uniform(-1.3, 1.2, (40, 2)),
                        C[-1] + rng.uniform(-0.2, 0.2, (8, 2)), C[:4], C[-2:] + [[0.15 + 1e-9, 0.0], [0.5 - 1e-7, 0.0]]])
    d = np.hypot(X[:, None, 0] - C[:, 0], X[:, None, 1] - C[:, 1])
    arcs = ((d < R + H) & (np.abs(d - R) < H)).sum(1)
    assert (arcs == 0).any() and (arcs == 1).any() and (arcs > 5).any()
    got = _wall(X, kernel)
    ref = O.to_world(Dk.disks_local_twelve(C, R, X, np.full(len(X), H), kernel), 0.0)
    scale = {"lam": 1.0, "G": H, "Cov": 1.0, "m1": 1 / H, "m2": 1 / H ** 2}
    for k in NAMES:
        assert np.abs(got[k] - ref[k]).max() * scale[k] <= 1e-10, k
    order = rng.permutation(len(X))
    many = _wall(np.concatenate([X[order], X[order][::-1]]), kernel)
    for k in NAMES:
        assert np.array_equal(many[k][: len(X)], got[k][order]) and np.array_equal(many[k][len(X):], got[k][order][::-1])
    for j in (int(np.argmax(arcs)), int(np.argmin(arcs)), len(X) - 1):
        one = _wall(X[j:j + 1], kernel)
        assert all(np.array_equal(one[k][0], got[k][j]) for k in NAMES)
