"""Launches of few rows with the workspace given as scratch (WSB_WS_SCRATCH): one kernel for the whole aggregate.

A block of it takes 16 to 128 consecutive rows, walks each row's pairs over the lanes of the sorted route and adds them in
its order, so every output must be the same bits as the sorted route's (tolerance 0), which is what the same call without
the flag runs; NaN stays NaN.  Sizes at the edges of a block and of a warp, with and without the allowed mask, adding
to outputs and assigning, over an unbounded body, for one kernel, a tensile one, a pack and a set that no pack covers.
Without the flag the workspace is left prepared: an evaluation on it gives the outputs again."""
import numpy as np
import pytest
import torch

from helpers import DEV, make_scene, small_c2
from warpsphboundaries_b200 import _lib
from warpsphboundaries_b200.kernels import KERNEL_IDS, QUAD_KERNEL_IDS
from warpsphboundaries_b200.scene import _stream

pytestmark = pytest.mark.gpu
IDS = {**KERNEL_IDS, **QUAD_KERNEL_IDS}
WIDTH = {"lam": (), "G": (2,), "Cov": (4,), "m1": (2,), "m2": (4,)}


def _call(loops, X, h, kernels, flags, precision=_lib.PREC_FP64, allowed=None, unbounded=0, after=False, background=0):
    scene, rep, body = make_scene(loops, center=(0.1, -0.3), angle=0.7, background=background)
    ns, n = rep.native(h, DEV), len(X)
    pos = torch.tensor(X, dtype=torch.float64, device=DEV)
    sup = torch.full((n,), h, dtype=torch.float64, device=DEV)
    al = None if allowed is None else torch.tensor(allowed, dtype=torch.int32, device=DEV)
    obb = (_lib.ctypes.c_double * 4)(*body.obb())
    ws, need = ns.workspace(n)
    out = [{k: torch.full((n,) + w, 0.25, dtype=torch.float64, device=DEV) for k, w in WIDTH.items()} for _ in kernels]
    ids, pose = _lib.int32s([IDS[k] for k in kernels]), body.pose_tensor(DEV)
    tgt = [_lib.ptrs([o[k] for o in out]) for k in WIDTH]
    _lib.check(_lib.lib.wsb_aggregate_groups(ns.handle, len(kernels), ids, precision, _lib.ptr(pos), _lib.ptr(sup),
                                             None if al is None else _lib.ptr(al), n, _lib.ptr(pose), obb, unbounded,
                                             _lib.OUT_ALL | flags, *tgt, _lib.ptr(ws), need, _stream()), "groups")
    got = [{k: v.cpu().numpy() for k, v in o.items()} for o in out]
    if not after:
        return got
    _lib.check(_lib.lib.wsb_aggregate_evaluate_groups(ns.handle, len(kernels), ids, precision, _lib.ptr(sup), n,
                                                      _lib.ptr(pose), _lib.OUT_ALL | flags, *tgt, _lib.ptr(ws), need,
                                                      _stream()), "evaluate")
    return got, [{k: v.cpu().numpy() for k, v in o.items()} for o in out]


def _same(a, b):
    return all(np.array_equal(x[k], y[k], equal_nan=True) for x, y in zip(a, b) for k in WIDTH)


def _rows(n):
    loops, X, h = small_c2()
    c, s = np.cos(0.7), np.sin(0.7)
    X = X[np.random.default_rng(n).integers(0, len(X), n)]
    return loops, X @ np.array([[c, s], [-s, c]]) + np.array([0.1, -0.3]), h


@pytest.mark.parametrize("n", [1, 15, 16, 17, 127, 128, 129, 4735, 4737, 40000])
def test_same_bits_as_the_sorted_rows(n):
    loops, X, h = _rows(n)
    allowed = np.random.default_rng(1).integers(0, 4, n) > 0
    for kernels in (("w4",), ("w2p5",), ("cubic", "w2", "w4", "w6"), ("cone", "quintic")):
        for flags, kw in ((_lib.OUT_ASSIGN, {}), (0, {}), (_lib.OUT_ASSIGN, {"allowed": allowed}), (0, {"allowed": allowed}),
                          (_lib.OUT_ASSIGN, {"unbounded": 1, "background": 1})):
            assert _same(_call(loops, X, h, kernels, flags | _lib.WS_SCRATCH, **kw), _call(loops, X, h, kernels, flags, **kw))


@pytest.mark.parametrize("precision", [_lib.PREC_MIXED, _lib.PREC_FP32])
def test_same_bits_in_the_other_precisions(precision):
    loops, X, h = _rows(700)
    for kernels in (("w4",), ("w2", "cone", "lw2")):
        a = _call(loops, X, h, kernels, _lib.OUT_ASSIGN | _lib.WS_SCRATCH, precision=precision)
        assert _same(a, _call(loops, X, h, kernels, _lib.OUT_ASSIGN, precision=precision))


def test_workspace_is_left_prepared_without_the_flag():
    loops, X, h = _rows(1000)
    got, again = _call(loops, X, h, ("w2", "w4", "w6"), _lib.OUT_ASSIGN, after=True)
    assert _same(got, again)


def _polygon(n, radius, h):
    """a wavy n-gon and its rms candidate-list length."""
    t = 2 * np.pi * np.arange(n) / n
    r = radius * (1 + 0.02 * np.sin(9 * t))
    P = np.stack([r * np.cos(t), r * np.sin(t)], 1)
    scene, rep, _ = make_scene([P], center=(0.1, -0.3), angle=0.7)
    length = np.diff(rep.native(h, DEV).cells()[0]).astype(float)
    return P, float(np.sqrt((length[length > 0] ** 2).mean()))


@pytest.mark.parametrize("edges,radius,h,n,kernels,one", [
    (256, 0.45, 0.03, 1 << 16, ("w4",), True), (256, 0.45, 0.03, 1 << 18, ("w4",), True),
    (600, 0.05, 0.1, 1 << 14, ("w4",), True), (600, 0.05, 0.1, 1 << 16, ("w4",), False),
    (1000, 0.2, 0.05, 1 << 16, ("w4",), False), (1000, 0.2, 0.05, 1 << 16, ("w2", "w4", "w6"), False),
    (256, 0.45, 0.03, 1 << 16, ("cubic", "w2", "w4", "w6"), True),
    (1000, 0.2, 0.05, 1 << 12, ("cubic", "w2", "w4", "w6"), True),
    (1000, 0.2, 0.05, 1 << 14, ("cubic", "w2", "w4", "w6"), False),
    (256, 0.2, 0.05, 1 << 17, ("w2p5",), False), (256, 0.45, 0.03, 1 << 17, ("w2p5",), True),
    (600, 0.3, 0.05, 1 << 15, ("w4", "cubic"), False), (600, 0.3, 0.05, 1 << 15, ("w4", "cone", "lw4"), True)])
def test_long_lists_go_to_the_sorted_rows(edges, radius, h, n, kernels, one):
    """the one-launch route leaves the workspace alone, the sorted route fills it: which of them a call takes follows its
    rows, its kernels and the length of the candidate lists; same bits either way."""
    P, length = _polygon(edges, radius, h)
    rng = np.random.default_rng(5)
    X = rng.uniform(-1.4 * radius - h, 1.4 * radius + h, (n, 2)) + np.array([0.1, -0.3])
    scene, rep, body = make_scene([P], center=(0.1, -0.3), angle=0.7)
    ns = rep.native(h, DEV)
    pos = torch.tensor(X, dtype=torch.float64, device=DEV)
    sup = torch.full((n,), h, dtype=torch.float64, device=DEV)
    obb, unbounded = body.broadphase()
    ws, need = ns.workspace(n)
    got = []
    for flags in (_lib.OUT_ASSIGN | _lib.WS_SCRATCH, _lib.OUT_ASSIGN):
        ws.fill_(0x5a)
        out = [{k: torch.empty((n,) + w, dtype=torch.float64, device=DEV) for k, w in WIDTH.items()} for _ in kernels]
        _lib.check(_lib.lib.wsb_aggregate_groups(
            ns.handle, len(kernels), _lib.int32s([IDS[k] for k in kernels]), _lib.PREC_FP64, _lib.ptr(pos), _lib.ptr(sup),
            None, n, _lib.ptr(body.pose_tensor(DEV)), obb, unbounded, _lib.OUT_ALL | flags,
            *[_lib.ptrs([o[k] for o in out]) for k in WIDTH], _lib.ptr(ws), need, _stream()), "groups")
        got.append((bool((ws == 0x5a).all()), out))
    assert (got[0][0], got[1][0]) == (one, False), length
    assert all(torch.equal(torch.nan_to_num(a[k]), torch.nan_to_num(b[k])) for a, b in zip(got[0][1], got[1][1]) for k in WIDTH)
