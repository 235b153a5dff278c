"""The radial family's two output paths -- the 28 baseline requests in their order, and any other set by its table -- at the
edges of a block of 128 rows, and the Gauss orders of every kernel against exact rational integration.

The two paths form each channel from the same invariants by the same products, so they agree within one rounding of a
product and a sum (4 ulp of the channel's terms)."""
import numpy as np
import pytest
import torch
from fractions import Fraction as F

from warpsphboundaries_b200 import kernels as K
from warpsphboundaries_b200.radial import RadialEvaluator, baseline

pytestmark = pytest.mark.gpu


def _rows(n, seed, h=0.05):
    rng = np.random.default_rng(seed)
    R = h * np.exp(rng.uniform(np.log(0.2), np.log(50.0), n))
    d = np.maximum(h * rng.uniform(-1.2, 1.2, n), -R)
    nrm = rng.normal(size=(n, 3))
    return d, nrm / np.linalg.norm(nrm, axis=1, keepdims=True), np.full(n, h), R


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000])
@pytest.mark.parametrize("kernel", ["cubic", "w2", "w4", "w6"])
def test_baseline_path_equals_the_table_path(n, kernel):
    d, nrm, h, R = _rows(n, n)
    full = RadialEvaluator("sphere", kernel=kernel)
    a = full.prepare(d, nrm, h, radii=R)
    a.launch()
    order = np.random.default_rng(1).permutation(28)
    b = RadialEvaluator("sphere", [baseline(3)[k] for k in order], kernel=kernel).prepare(d, nrm, h, radii=R)
    b.launch()
    c = RadialEvaluator("sphere", baseline(3)[:1], kernel=kernel).prepare(d, nrm, h, radii=R)
    c.launch()
    va, vb = a.values.cpu().numpy(), b.values.cpu().numpy()
    scale = np.abs(va).max(axis=0) + 1e-300
    assert (np.abs(va[:, order] - vb) <= 4 * 2.0 ** -52 * scale[order]).all()
    assert torch.equal(c.values[:, 0], a.values[:, 0]) and torch.equal(a.work, b.work) and torch.equal(a.work, c.work)
    assert int(a.status.abs().sum()) == 0 and np.isfinite(va).all()


@pytest.mark.parametrize("kernel", ["cubic", "w2", "w4", "w6"])
def test_half_space_mass_is_exact(kernel):
    """lam of a half-space: the exact polynomial in d, from the rational tables (d on the dyadic grid): 1e-14."""
    ds = [F(k, 16) for k in range(-16, 17)]
    ref = []
    pcs, _ = K.radial(kernel)
    for d in ds:
        tot = F(0)
        for lo, hi, W, _, _ in pcs:
            poly = K._pmul(list(W.g), K._ppow([hi, F(-1)], W.k)) if W.k else list(W.g)
            ball, cap = (lo, min(hi, max(F(0), -d))), (max(lo, abs(d)), hi)
            for (a, b), f in ((ball, [F(0), F(0), F(4)]), (cap, [F(0), -2 * d, F(2)])):     # r^2 a0 = 4 r^2 and 2 r (r - d)
                if b > a:
                    q = K._pmul(poly, f)
                    tot += sum(c * (b ** (k + 1) - a ** (k + 1)) / (k + 1) for k, c in enumerate(q))
        ref.append(float(tot))
    ev = RadialEvaluator("plane", baseline(3)[:1], kernel=kernel)
    got = ev.evaluate(np.array([float(d) for d in ds]), np.tile([0.0, 0.0, 1.0], (len(ds), 1)), 1.0)
    assert np.abs(got[:, 0] - np.array(ref)).max() <= 1e-14
