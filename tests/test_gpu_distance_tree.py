"""The edge tree of the signed distance at the sizes where its levels change (8 edges a leaf, 8 nodes a node): distance,
closest point and edge equal a scan over all edges in the same rounded operations -- exactly, the lower id on a tie --
for points near, far outside the grid, on vertices and at equal distance to two edges; and the one-pass form over posed
bodies equals the composition of the frame changes, exactly."""
import numpy as np
import pytest
import torch

from oracle import edge2d as O
from warpsphboundaries_b200 import _lib, workloads
from warpsphboundaries_b200.scene import Body, Scene, SurfaceRep, _stream

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _distance(ns, P, support):
    m = len(P)
    lp = torch.tensor(P, dtype=torch.float64, device=DEV)
    d = torch.empty(m, dtype=torch.float64, device=DEV)
    cp, nl = (torch.empty((m, 2), dtype=torch.float64, device=DEV) for _ in range(2))
    ed = torch.empty(m, dtype=torch.int32, device=DEV)
    _lib.check(_lib.lib.wsb_signed_distance(ns.handle, _lib.ptr(lp), m, support, _lib.ptr(d), _lib.ptr(cp), _lib.ptr(nl),
                                            _lib.ptr(ed), _stream()), "wsb_signed_distance")
    return [t.cpu().numpy() for t in (d, cp, nl, ed)]


def _scan(V, E, P):
    """numpy rounds every operation: the order of the operations is the kernel's."""
    a, b = V[E[:, 0]], V[E[:, 1]]
    e = b - a
    best, cp, ed = np.full(len(P), np.inf), np.zeros((len(P), 2)), np.full(len(P), -1)
    for k in range(len(E)):
        t = ((P[:, 0] - a[k, 0]) * e[k, 0] + (P[:, 1] - a[k, 1]) * e[k, 1]) / (e[k, 0] * e[k, 0] + e[k, 1] * e[k, 1])
        t = np.clip(t, 0.0, 1.0)
        c = np.stack([a[k, 0] + t * e[k, 0], a[k, 1] + t * e[k, 1]], 1)
        dist = np.sqrt((P[:, 0] - c[:, 0]) ** 2 + (P[:, 1] - c[:, 1]) ** 2)
        near = dist < best
        best[near], cp[near], ed[near] = dist[near], c[near], k
    return best, cp, ed


@pytest.mark.parametrize("n", [3, 8, 9, 64, 65, 512, 513, 1500])
def test_tree_equals_the_scan(n):
    rng = np.random.default_rng(n)
    loop = workloads.star(rng, (0.2, -0.1), 0.5, n)
    rep = SurfaceRep.polygon(loop, conditioned=False)
    V, E = rep.vertices.numpy(), rep.edges.numpy().astype(np.int64)
    P = np.concatenate([rng.uniform(-0.6, 0.9, (600, 2)), rng.uniform(-40.0, 40.0, (60, 2)), V[: min(n, 40)],
                        0.5 * (V[: min(n, 40)] + V[(np.arange(min(n, 40)) + 1) % n]), [[0.2, -0.1]]])
    d, cp, nl, ed = _distance(rep.native(0.03, DEV), P, 0.03)
    best, c, k = _scan(V, E, P)
    assert np.array_equal(np.abs(d), best)
    assert np.array_equal(cp, c) and np.array_equal(ed, k)
    off = best > 1e-9
    assert np.array_equal(d[off] < 0, O.indicator(V, E, 0, P[off]) > 0.5)


def test_posed_bodies_in_one_pass():
    rng = np.random.default_rng(3)
    tank = workloads.star(rng, (0.0, 0.0), 3.0, 48, jitter=0.0)
    bodies = [Body(reps=[SurfaceRep.polygon(tank, "outside")])]
    for k in range(3):
        loops = [workloads.star(rng, (0.0, 0.0), 0.3, 40 + k), workloads.star(rng, (0.7, 0.0), 0.2, 20)]
        bodies.append(Body(center=tuple(rng.uniform(-1.5, 1.5, 2)), angle=float(rng.uniform(-3, 3)),
                           reps=[SurfaceRep.polygon(p) for p in loops]))
    scene = Scene(bodies, DEV)
    P = torch.tensor(rng.uniform(-3.5, 3.5, (4000, 2)), device=DEV)
    for only in (None, 2):
        d, n, hit, b = scene.signed_distance(P, body=only, supportMax=0.05, want_body=True)
        best = torch.full((len(P),), float("inf"), dtype=torch.float64, device=DEV)
        normal, index = torch.zeros_like(P), torch.full((len(P),), -1, dtype=torch.long, device=DEV)
        for bi, body in enumerate(scene.bodies):
            for rep in body.reps if only in (None, bi) else ():
                lp = body.toLocal(P).contiguous().cpu().numpy()
                dd, _, nl, _ = (torch.tensor(t, device=DEV) for t in _distance(rep.native(0.05, DEV), lp, 0.05))
                better = dd < best
                best = torch.where(better, dd, best)
                normal = torch.where(better[:, None], body.pose.vecToWorld(nl), normal)
                index = torch.where(better, torch.full_like(index, bi), index)
        assert torch.equal(d, best) and torch.equal(n, normal) and torch.equal(b, index) and bool(hit.all())
    d, n, hit, b = Scene([Body()], DEV).signed_distance(P, want_body=True)
    assert bool(torch.isinf(d).all()) and not bool(n.any()) and not bool(hit.any()) and bool((b == -1).all())
