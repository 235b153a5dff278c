"""Derivatives of Scene.signed_distance by the points: the analytic shapes (disk, box) are differentiable, the polygonal
surfaces' rows have none -- whatever the order of the bodies, in reverse and in forward mode."""
import numpy as np
import pytest
import torch
import torch.autograd.forward_ad as fwAD

from warpsphboundaries_b200 import workloads
from warpsphboundaries_b200.implicit import DiskBody
from warpsphboundaries_b200.scene import Body, BoxRep, ImplicitRep, Scene, SurfaceRep

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _bodies():
    rng = np.random.default_rng(2)
    star = SurfaceRep.polygon(workloads.star(rng, (0.0, 0.0), 0.4, 40), conditioned=False)
    return {"star": Body(center=(-0.5, 0.1), angle=0.4, reps=[star]),
            "disk": Body(center=(0.6, -0.2), reps=[ImplicitRep(DiskBody((0.0, 0.0), 0.3))]),
            "box": Body(center=(0.1, 0.9), angle=0.2, reps=[BoxRep((-0.2, -0.1), (0.3, 0.2))])}


@pytest.mark.parametrize("order", [("disk", "star"), ("star", "disk"), ("disk", "star", "box"), ("box", "disk", "star")])
def test_derivative_of_the_nearest_shape(order):
    bodies = _bodies()
    scene = Scene([bodies[k] for k in order], DEV)
    rng = np.random.default_rng(9)
    X = torch.tensor(rng.uniform(-1.4, 1.4, (3000, 2)), device=DEV)
    plain, normal, _, index = scene.signed_distance(X, supportMax=0.1, want_body=True)
    surface = index == order.index("star")
    assert 300 < int(surface.sum()) < 2700
    P = X.clone().requires_grad_()
    d, n, _, b = scene.signed_distance(P, supportMax=0.1, want_body=True)
    assert torch.equal(d, plain) and torch.equal(n, normal) and torch.equal(b, index)
    (g,) = torch.autograd.grad(d.sum() + (n * torch.tensor([0.3, -0.7], device=DEV)).sum(), P, retain_graph=True)
    assert not bool(g[surface].any())
    (g,) = torch.autograd.grad(d.sum(), P)
    want = torch.where(surface[:, None], torch.zeros_like(normal), normal)
    kinks = (g - want).abs().amax(1) > 1e-9                    # inside the box: the faces' normals, not the closest point's
    assert int(kinks.sum()) == 0
    with fwAD.dual_level():
        d, n, _ = scene.signed_distance(fwAD.make_dual(X, torch.ones_like(X)), supportMax=0.1)
        assert torch.equal(d.detach(), plain)
        tangent = fwAD.unpack_dual(d).tangent
    assert float((tangent - want.sum(1)).abs().max()) <= 1e-9
