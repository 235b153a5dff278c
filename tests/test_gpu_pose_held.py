"""A wall evaluation and a signed distance hold the device pose they hand to the library until their calls are made,
whatever becomes of the body's own cached copy meanwhile (another thread moving the body, another scene asking for it on
another device)."""
import weakref

import numpy as np
import pytest
import torch

from warpsphboundaries_b200 import provider, workloads
from warpsphboundaries_b200 import scene as scene_module
from warpsphboundaries_b200.provider import FusedGroup, FusedWall
from warpsphboundaries_b200.scene import Body, DiskArrayRep, Scene, SurfaceRep
from warpsphboundaries_b200.shim import ParticleState

pytestmark = pytest.mark.gpu


def test_pose_outlives_the_cache(monkeypatch):
    rng = np.random.default_rng(1)
    reps = [SurfaceRep.polygon(workloads.star(rng, (k, 0.0), 0.3, 40), conditioned=False) for k in (0.0, 1.0)]
    body = Body(center=(0.2, 0.1), angle=0.4, reps=reps + [DiskArrayRep([[0.0, 1.0]], [0.2])])
    scene = Scene([body], "cuda")
    pos = torch.tensor(rng.uniform(-1.0, 2.0, (2000, 2)), device="cuda")
    ps = ParticleState(pos, torch.full((2000,), 0.1, dtype=torch.float64, device="cuda"))
    dist = scene.signed_distance(pos, supportMax=0.1)
    want = {k: v.clone() for k, v in FusedWall(scene, ps, 0.1, (FusedGroup("w4"),)).res[0].items()}
    seen, calls = [], []
    form = Body.pose_tensor

    def replaced(self, device):
        t = form(self, device).clone()
        self.__dict__.pop("_poseCache", None)          # the body keeps nothing
        seen.append(weakref.ref(t))
        return t

    class Library:
        def __getattr__(self, name):
            f = getattr(provider._lib.lib, name)
            if name not in ("wsb_aggregate_groups", "wsb_disk_aggregate", "wsb_body_distance"):
                return f

            def call(*a):
                calls.append(seen[-1]() is not None)
                return f(*a)
            return call

    monkeypatch.setattr(Body, "pose_tensor", replaced)
    monkeypatch.setattr(provider, "lib", Library())
    monkeypatch.setattr(scene_module, "lib", Library())
    got = FusedWall(scene, ps, 0.1, (FusedGroup("w4"),)).res[0]
    assert calls == [True, True, True]
    assert all(torch.equal(got[k], want[k]) for k in want)
    again = scene.signed_distance(pos, supportMax=0.1)
    assert calls == [True] * 5
    assert all(torch.equal(a, b) for a, b in zip(again, dist))
