"""A body that a call has used (its box cached as C doubles, its device pose cached) is copied and pickled like a new one."""
import copy
import pickle

import torch

from warpsphboundaries_b200 import _lib
from warpsphboundaries_b200.scene import Body, SurfaceRep


def test_used_body_is_copied_and_pickled():
    body = Body(center=(0.25, -1.0), angle=0.3,
                reps=[SurfaceRep.loops([[[0.0, 0.0], [1.0, 0.0], [0.0, 1.0]]], solid="inside")])
    box, unbounded = body.broadphase()
    pose = body.pose_tensor(torch.device("cpu"))
    assert isinstance(box, _lib.ctypes.Array) and tuple(box) == body.obb()
    for other in (copy.copy(body), copy.deepcopy(body), pickle.loads(pickle.dumps(body))):
        again, flag = other.broadphase()
        assert tuple(again) == tuple(box) and flag == unbounded
        assert torch.equal(other.pose_tensor(torch.device("cpu")), pose)
    _lib.POINTER(_lib.c_double).from_param(box)          # what the entry points take
