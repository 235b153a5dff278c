"""The (row, face) pair queue of the closed-surface evaluation: a warp integrates 32 pairs at a time, whatever rows they
belong to, so a row's faces may fill part of a round, exactly one, or several.

Rows with no face, one face, around 32 and 64 faces and several hundred, alone and among others: the same bits.  Values
against the oracle within 1e-10 (1 + max |v|) in units of the support (gradients times h, the Hessian times h^2): the
potentials' monomial form loses sum |c_n| / max |A| (at most about 2e5, for w6) units of 2^-53, and a few hundred such
terms add up."""
import numpy as np
import pytest
import torch

from oracle import mesh3d as M3
from warpsphboundaries_b200 import workloads as W
from warpsphboundaries_b200.mesh3d import ClosedMesh

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


def _channels(mesh, Q, h, kernel):
    out = mesh.channels(torch.tensor(Q, dtype=torch.float64, device=DEV), torch.tensor(h, dtype=torch.float64, device=DEV),
                        kernel)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _unit(v, h):
    """channels in units of the support: value moments by h^-|alpha|, gradient moments and the Hessian likewise."""
    p = np.concatenate([[0], np.full(3, -1), np.full(6, -2), np.full(3, 1), np.zeros(9), np.full(6, 2)])
    return v * h ** p


def _faces_within(V, Fc, q, h):
    """an upper estimate of the row's faces: those with a sampled point within h."""
    b = np.array([(i / 8, j / 8, 1 - i / 8 - j / 8) for i in range(9) for j in range(9 - i)])
    pts = np.einsum("bk,fkd->fbd", b, V[Fc])
    return int((np.linalg.norm(pts - q, axis=2).min(1) < h).sum())


@pytest.mark.parametrize("kernel", ["cubic", "w2", "w4", "w6"])
def test_rows_of_every_face_count(kernel):
    V, Fc = W.icosphere(3, 0.6, 0.05, seed=4)                     # 1280 faces
    rng = np.random.default_rng(12)
    Q, h = [], []
    for hh in (0.02, 0.05, 0.1, 0.13, 0.18, 0.25, 0.35):
        d = rng.normal(size=(5, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        Q.append(d * (0.6 + hh * rng.uniform(-0.9, 0.9, (5, 1))))
        h.append(np.full(5, hh))
    Q, h = np.concatenate(Q), np.concatenate(h)
    counts = [_faces_within(V, Fc, q, s) for q, s in zip(Q, h)]
    assert min(counts) <= 2 and max(counts) > 128 and any(24 <= c <= 40 for c in counts)
    mesh = ClosedMesh(V, Fc, 0.35, DEV)
    together = _channels(mesh, Q, h, kernel)
    order = rng.permutation(len(Q))
    shuffled = _channels(mesh, np.repeat(Q[order], 3, 0), np.repeat(h[order], 3), kernel)
    for k in range(len(Q)):
        assert np.array_equal(_channels(mesh, Q[k:k + 1], h[k:k + 1], kernel)[0], together[k]), k
    assert np.array_equal(shuffled, np.repeat(together[order], 3, 0))
    for k in range(0, len(Q), 5):
        ref = _unit(M3.channels(V, Fc, Q[k], h[k], kernel), h[k])
        assert np.abs(_unit(together[k], h[k]) - ref).max() <= 1e-10 * (1 + np.abs(ref).max()), (k, counts[k])


@pytest.mark.parametrize("kernel", ["cubic", "w6"])
def test_short_edges_and_planes_through_the_query(kernel):
    """faces far smaller than the support (edges of 1/40 h) and queries in the plane, on an edge line or on a vertex
    ray of a box's faces."""
    V, Fc = W.icosphere(4, 0.6, 0.02, seed=6)                     # edges of about 0.04
    Q = np.array([[0.31, 0.2, 0.4]])
    h = np.full(len(Q), 0.5)
    got = _channels(ClosedMesh(V, Fc, 0.5, DEV), Q, h, kernel)
    Vb, Fb = W.box_mesh((-0.3, -0.25, -0.2), (0.35, 0.3, 0.25))
    Qb = np.array([[0.4, 0.1, 0.25], [0.35 + 1e-9, 0.3 + 1e-9, 0.1], [0.45, 0.3, 0.25], [0.36, 0.31, 0.26], [0.3, 0.3, 0.3]])
    hb = np.full(len(Qb), 0.2)
    gotb = _channels(ClosedMesh(Vb, Fb, 0.2, DEV), Qb, hb, kernel)
    for V_, F_, Q_, h_, g_ in ((V, Fc, Q, h, got), (Vb, Fb, Qb, hb, gotb)):
        for k in range(len(Q_)):
            ref = _unit(M3.channels(V_, F_, Q_[k], h_[k], kernel), h_[k])
            assert np.abs(_unit(g_[k], h_[k]) - ref).max() <= 1e-9 * (1 + np.abs(ref).max()), k


@pytest.mark.parametrize("kernel", ["cubic", "w2", "w4", "w6"])
def test_a_vertex_just_inside_the_support(kernel):
    """faces that reach into the support by a vertex only, by 1e-7 to 1e-9 supports, the foot of the query outside them:
    the edges' angles beyond the support are of order one and cancel to the angle of that depth."""
    rng = np.random.default_rng(21)
    apex, axis = np.array([0.1, -0.2, 0.05]), np.array([0.48, 0.6, 0.64])
    base = np.linalg.svd(axis[None])[2][1:]                      # two directions across the axis
    ring = [0.2 * (np.cos(t) * base[0] + np.sin(t) * base[1]) for t in (0.3, 2.1, 4.6)]
    V = np.concatenate([[apex], apex - axis * np.array([[0.25], [0.4], [0.3]]) + ring])
    Fc = np.array([[0, 1, 2], [0, 2, 3], [0, 3, 1], [1, 3, 2]])
    if np.dot(np.cross(V[1] - V[0], V[2] - V[0]), V[3] - V[0]) > 0:
        Fc = Fc[:, ::-1].copy()                                  # outward normals
    u = axis + rng.uniform(0.3, 1.2, (24, 1)) * _directions(rng, 24, base)
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    Q = np.concatenate([apex + (1.0 - depth) * u for depth in (1e-7, 1e-8, 1e-9)])
    h = np.ones(len(Q))
    got = _channels(ClosedMesh(V, Fc, 1.0, DEV), Q, h, kernel)
    for k in range(len(Q)):
        ref = M3.channels(V, Fc, Q[k], 1.0, kernel)
        assert np.abs(got[k] - ref).max() <= 1e-10 * (1 + np.abs(ref).max()), k


def _directions(rng, n, base):
    t = rng.uniform(0, 2 * np.pi, n)
    return np.cos(t)[:, None] * base[0] + np.sin(t)[:, None] * base[1]
