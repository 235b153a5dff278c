"""The lane splits of the 2-D wall pass: rows of many pairs (two lanes a row, eight from 32 pairs on, from 16 on for the
tensile kernels), cells of long candidate lists (eight lanes a row) and the lanes of the other rows by the launch's size,
with candidates past the 128 of a row's mask.

A polygon of edges far shorter than the support gives rows of 0 to some 250 pairs, every count around the limits among
them.  Against the oracle within 1e-10 in units of the support (the tolerance of the parity tests); a row's bits do not
depend on how many rows are launched with it."""
import numpy as np
import pytest
import torch

from oracle import edge2d as O
from tests.helpers import DEV, gpu_outputs, make_scene, oracle_outputs, scaled_errors
from warpsphboundaries_b200 import workloads

pytestmark = pytest.mark.gpu
H = 0.05


def _scene():
    """a fine ring (edges of H / 120, then H / 8 and H / 3 sectors) and a coarse square."""
    t = np.concatenate([np.linspace(0, 2.0, 2400, endpoint=False), np.linspace(2.0, 4.0, 160, endpoint=False),
                        np.linspace(4.0, 2 * np.pi, 70, endpoint=False)])
    ring = np.stack([0.5 * np.cos(t), 0.5 * np.sin(t)], 1)
    return [ring, np.array([[0.8, -0.2], [1.2, -0.2], [1.2, 0.2], [0.8, 0.2]])]


def _rows(n, seed):
    rng = np.random.default_rng(seed)
    a = rng.uniform(0, 2 * np.pi, n)
    r = 0.5 + H * rng.uniform(-1.1, 1.1, n)
    X = np.stack([r * np.cos(a), r * np.sin(a)], 1)
    X[: n // 10] = rng.uniform(-0.7, 1.4, (n // 10, 2))
    return X


def _counts(loops, X):
    V, E = workloads.edges_of(loops)
    a, d = V[E[:, 0]], V[E[:, 1]] - V[E[:, 0]]
    t = np.clip(((X[:, None] - a) * d).sum(2) / (d * d).sum(1), 0, 1)
    return (np.linalg.norm(X[:, None] - a - t[..., None] * d, axis=2) < H).sum(1)


@pytest.mark.parametrize("kernel", ["w4", "cubic"])
def test_rows_of_every_pair_count(kernel):
    loops, X = _scene(), _rows(700, 3)
    c = _counts(loops, X)
    assert {0, 15, 16, 17}.issubset(c) and (c > 128).any() and any(k in c for k in (31, 32, 33))
    scene, _, _ = make_scene(loops, center=(0.1, -0.2), angle=0.4)
    W = X @ np.array([[np.cos(0.4), np.sin(0.4)], [-np.sin(0.4), np.cos(0.4)]]) + np.array([0.1, -0.2])
    got = gpu_outputs(scene, W, H, kernel, H)
    ref = oracle_outputs(loops, W, H, kernel, H, center=(0.1, -0.2), angle=0.4)
    assert max(scaled_errors(got, ref, H).values()) <= 1e-10
    # the same rows inside launches of every lane choice, and alone
    for n in (1, 60000, 300000, 600000):
        Y = W[:1] if n == 1 else np.concatenate([W, _rows(n - len(W), 5)])
        more = gpu_outputs(scene, Y, H, kernel, H)
        k = min(len(W), len(Y))
        assert all(np.array_equal(more[q][:k], got[q][:k]) for q in got)


@pytest.mark.parametrize("kernel", ["w2p5", "w4p5"])
def test_tensile_rows_of_every_pair_count(kernel):
    loops, X = _scene(), _rows(500, 9)
    V, E = workloads.edges_of(loops)
    scene, _, _ = make_scene(loops)
    G = gpu_outputs(scene, X, H, kernel, H)["G"]
    pick = np.argsort(_counts(loops, X))[::12]
    ref = O.powered_gradient_local(V, E, X[pick], H, kernel)
    assert np.abs((G[pick] - ref) * H).max() <= 1e-10
    again = gpu_outputs(scene, np.concatenate([_rows(1000, 2), X]), H, kernel, H)["G"][1000:]
    assert np.array_equal(again, G)
