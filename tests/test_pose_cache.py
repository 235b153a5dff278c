"""A body's device pose follows its centre: another centre tensor may lie in the memory of an earlier one."""
import numpy as np
import torch

from warpsphboundaries_b200.scene import Body, SurfaceRep


def test_pose_follows_replaced_and_changed_centres():
    body = Body(angle=0.3, reps=[SurfaceRep.loops([[[0.0, 0.0], [1.0, 0.0], [0.0, 1.0]]], solid="inside")])
    dev, where = torch.device("cpu"), np.zeros(2)
    for k in range(3):
        where[:] = (k, -2.0 * k)               # a host program's own array, wrapped anew each step
        body.center = torch.from_numpy(where)
        assert torch.equal(body.pose_tensor(dev)[:2], torch.tensor([k, -2.0 * k], dtype=torch.float64))
    held = body.pose_tensor(dev)
    assert body.pose_tensor(dev) is held       # unchanged: the same tensor
    body.center.add_(1.0)
    assert torch.equal(body.pose_tensor(dev)[:2], body.center)
