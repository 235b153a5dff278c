"""The float32 half-space and sphere invariants: no further from the float64 values than a float32 sum over twelve nodes a
region on the host (numpy, every operation rounded to float32, products added fused), the Hessian's two terms, which
cancel, combined at the node.  The tolerance of 1.15 on the root mean square covers the order of the operations; fewer
nodes, or sums of the two terms apart, give 1.2 to 1.4."""
import numpy as np
import pytest
import torch

from warpsphboundaries_b200 import kernels as K
from warpsphboundaries_b200.radial import RadialEvaluator

pytestmark = pytest.mark.gpu
f32, f64 = np.float32, np.float64


def _fma(a, b, c):
    return (np.asarray(a, f64) * np.asarray(b, f64) + np.asarray(c, f64)).astype(f32)


def _profile(f, hi, r):
    g = np.full_like(r, f32(f.g[-1]))
    for c in list(f.g)[-2::-1]:
        g = _fma(g, r, f32(c))
    for _ in range(abs(f.p)):
        g = g * r if f.p > 0 else g / r
    for _ in range(f.k):
        g = g * (f32(hi) - r)
    return g


def _host(d, R, kernel):
    """the nine invariants of the partial caps and full balls, unit support, float32."""
    x, w = np.polynomial.legendre.leggauss(12)
    out = np.zeros((len(d), 9), f32)
    pieces, _ = K.radial(kernel)
    third = f32(1.0 / 3.0)
    for lo, hi, W, L, dL in pieces:
        for full in (True, False):
            a = np.full_like(d, f32(lo)) if full else np.maximum(f32(lo), np.abs(d))
            b = np.minimum(f32(hi), np.clip(-d, 0, 1) if full else (np.ones_like(d) if R is None
                                                                    else np.minimum(f32(1), f32(2) * R + d)))
            on = (b > a) & (d > -1) & (d < 1)
            c, hw = f32(0.5) * (b + a), f32(0.5) * (b - a)
            s = np.zeros((9, len(d)), f32)
            for xg, wg in zip(x.astype(f32), w.astype(f32)):
                r = _fma(hw, xg, c)
                with np.errstate(all="ignore"):
                    v, l, dl = (_profile(f, hi, r) for f in (W, L, dL))
                if full:
                    r2 = wg * r * r
                    q4, q43 = f32(4), f32(4.0 / 3.0)
                    hes = _fma(q4 * r2, l, (q43 * (r2 * r)) * dl)
                    terms = (q4 * r2 * v, 0, q43 * (r2 * r * r) * v, q43 * (r2 * r * r) * v, 0, -q43 * (r2 * r * r) * l,
                             -q43 * (r2 * r * r) * l, hes, hes)
                else:
                    ru, rv = r - d, r + d
                    if R is not None:
                        i2 = f32(1) / (f32(2) * (R + d))
                        ru, rv = ru * (((R - r) + (R + d)) * i2), rv * ((rv + f32(2) * R) * i2)
                    rc = f32(0.5) * (ru - rv)
                    a1, at, an = ru * rv, ru * ru * (r + rv), ru * _fma(rc, rc - r, r * r)
                    wr = wg * r
                    lu, wd = wr * l * ru, wg * f32(1.0 / 6.0) * dl
                    terms = (f32(2) * (wr * v) * ru, -(wr * v) * a1, third * ((wr * v) * at), f32(2) * third * ((wr * v) * an),
                             (wr * l) * a1, -third * ((wr * l) * at), -f32(2) * third * ((wr * l) * an),
                             f32(2) * _fma(wd, at, lu), f32(2) * _fma(f32(2) * wd, an, lu))
                for j, t in enumerate(terms):
                    s[j] = s[j] + t
            out[on] += (hw * s).T[on]
    return out


@pytest.mark.parametrize("kind", ["plane", "sphere"])
@pytest.mark.parametrize("kernel", ["cubic", "w2", "w4", "w6"])
def test_rms_error_of_twelve_nodes(kind, kernel):
    rng = np.random.default_rng(31)
    n = 8000
    R = np.exp(rng.uniform(np.log(0.02), np.log(50.0), n)).astype(f32)
    d = np.maximum(rng.uniform(-0.98, 0.98, n).astype(f32), -R * f32(0.98))
    nrm = rng.normal(size=(n, 3))
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    dev = lambda t: torch.tensor(np.asarray(t, f64), device="cuda")
    got = []
    for precision in ("float32", "float64"):
        b = RadialEvaluator(kind, kernel=kernel, precision=precision).prepare(
            dev(d), dev(nrm), dev(np.ones(n)), **({"radii": dev(R)} if kind == "sphere" else {}))
        b.launch()
        got.append(b.work.double().cpu().numpy())
    host = _host(d, R if kind == "sphere" else None, kernel)
    assert np.abs(host - got[1]).max() < 1e-4                    # the same integrals
    rms = [float(np.sqrt(np.mean((v - got[1]) ** 2))) for v in (got[0], host.astype(f64))]
    assert rms[0] <= 1.15 * rms[1], rms
