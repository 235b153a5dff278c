"""The calls that users of this package make in earnest, as cases that can be timed and checked one by one.

`listed()` gives them, `draw(rng)` more of the same ranges.  `prepare(case, seed)` is what a program holds before the
call (inputs, scene, evaluator), `run(state)` one pass through the public entry points, `work(case)` the bytes and
float64 operations that the pass cannot do without, and `exact(case, seed)` the same outputs from plain torch in float64
(brute-force neighbours, adaptive panels of Gauss-Legendre nodes; none of the package's kernels).

Families (`what`):
  wall       AnalyticBoundary.aggregate(lean=True) at the particles of one scene: lambda, G, Cov, m1, m2 (a scheme's call
             once per time step and kernel)
  groups     FusedWall with several smoothing kernels at one position set (a convergence or a kernel study)
  delta      AnalyticBoundary.aggregate without `lean` and with the wall Laplacian: the delta+ scheme's call
  bodies     aggregate in a tank with several posed bodies ([B, N] outputs)
  adjoint    autograd through aggregate_moments: forward and gradients to particles and vertices
  distance   AnalyticBoundary.signed_distance (shifting, wall functions, initial packing)
  disks      aggregate of a fibre bundle (DiskArrayRep)
  mesh       Evaluator over Geometry.closed_surface: the 28 channels of a closed triangle surface
  spheres    RadialEvaluator("sphere"): the 28 channels of solid spheres, one row per (query, sphere)
  planes     RadialEvaluator("plane"): half-spaces
"""
import math
from fractions import Fraction as F

import numpy as np
import torch

F64 = torch.float64
DEV = "cuda"

KERNELS = ("cubic", "w2", "w4", "w6")
SCHEME = {"cubic": "CubicSpline", "w2": "Wendland2", "w4": "Wendland4", "w6": "Wendland6"}
STARS = {"stars": 64, "vmin": 32, "vmax": 512}


# ------------------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one small tank of a unit test or an interactive run: latency and launches count
        {"name": "wall_4k", "what": "wall", "n": 4096, "kernel": "w4", "shape": "gon", "h": 0.05},
        # a production step: 2^20 particles among 64 polygons
        {"name": "wall_1m", "what": "wall", "n": 1 << 20, "kernel": "w4", "shape": "stars", "h": 0.02},
        # the four smoothing kernels at once on the same scene (the benchmark's step)
        {"name": "groups_1m", "what": "groups", "n": 1 << 20, "kernels": "cubic,w2,w4,w6", "h": 0.02},
        # the delta+ scheme's wall evaluation: scheme kernel, cover vector, wall Laplacian, tensile kernel; odd count
        {"name": "delta_300k", "what": "delta", "n": 300001, "kernel": "w2", "h": 0.02},
        # moving bodies in a tank, supports that differ from particle to particle
        {"name": "bodies_65k", "what": "bodies", "n": 65537, "kernel": "w2", "bodies": 8, "h": 0.02},
        # differentiable simulation: gradients to 2^18 particles and to the vertices of 16 polygons
        {"name": "adjoint_262k", "what": "adjoint", "n": 1 << 18, "kernel": "w4", "h": 0.02},
        # signed distance and normal of every particle
        {"name": "distance_200k", "what": "distance", "n": 200003, "h": 0.02},
        # a bundle of 1024 fibres
        {"name": "disks_1m", "what": "disks", "n": 1 << 20, "kernel": "w4", "disks": 1024, "h": 0.02},
        # the particles next to a closed surface, as a 3-D solver queries it
        {"name": "mesh_near_20k", "what": "mesh", "n": 20011, "kernel": "w2", "subdivisions": 5, "h": 0.03, "near": True},
        # every particle of a 3-D domain against a surface of 20480 faces
        {"name": "mesh_2m", "what": "mesh", "n": 1 << 21, "kernel": "w4", "subdivisions": 5, "h": 0.03, "near": False},
        # a few thousand rows of half-spaces (a flat floor)
        {"name": "planes_10k", "what": "planes", "n": 10007, "kernel": "w2", "h": 0.03},
        # 2^21 rows of solid spheres with radii from 0.2 to 50 supports
        {"name": "spheres_2m", "what": "spheres", "n": 1 << 21, "kernel": "w4", "h": 0.03},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1

    what = rng.choice(("wall", "wall", "groups", "delta", "bodies", "adjoint", "distance", "disks", "mesh", "mesh",
                       "spheres", "planes"))
    kernel = rng.choice(KERNELS)
    if what == "wall":
        shape = rng.choice(("gon", "stars"))
        h = rng.uniform(0.02, 0.08) if shape == "gon" else rng.uniform(0.01, 0.03)
        return {"what": what, "n": size(1000, 1 << 20), "kernel": kernel, "shape": shape, "h": round(h, 4)}
    if what == "groups":
        sets = ("w2,w4,w6", "cubic,w2,w4,w6", "w4,cubic", "w6,w2")
        return {"what": what, "n": size(2000, 1 << 20), "kernels": rng.choice(sets), "h": round(rng.uniform(0.01, 0.025), 4)}
    if what == "delta":
        return {"what": what, "n": size(2000, 1 << 19), "kernel": rng.choice(("w2", "w4")),
                "h": round(rng.uniform(0.01, 0.025), 4)}
    if what == "bodies":
        return {"what": what, "n": size(1000, 1 << 18), "kernel": kernel, "bodies": rng.randint(2, 12),
                "h": round(rng.uniform(0.01, 0.03), 4)}
    if what == "adjoint":
        return {"what": what, "n": size(1000, 1 << 19), "kernel": kernel, "h": round(rng.uniform(0.01, 0.03), 4)}
    if what == "distance":
        return {"what": what, "n": size(1000, 1 << 18), "h": round(rng.uniform(0.015, 0.03), 4)}
    if what == "disks":
        return {"what": what, "n": size(2000, 1 << 20), "kernel": kernel, "disks": rng.randint(1, 1024),
                "h": round(rng.uniform(0.01, 0.03), 4)}
    if what == "mesh":
        near = rng.random() < 0.5
        return {"what": what, "n": size(1000, 20000) if near else size(1000, 1 << 20), "kernel": kernel,
                "subdivisions": rng.choice((3, 4, 5)), "h": round(rng.uniform(0.02, 0.06 if not near else 0.04), 4),
                "near": near}
    return {"what": what, "n": size(1000, 1 << 21), "kernel": kernel, "h": round(rng.uniform(0.01, 0.1), 4)}


# ------------------------------------------------------------------------------------------------------------ the inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _stars(seed, count, vmin, vmax, box=4.0, rmin=0.05, rmax=0.4):
    """star polygons [n, 2], counter-clockwise: centre uniform, mean radius log-uniform, radial jitter +-15 %."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(count):
        c, n = rng.uniform(0, box, 2), int(rng.integers(vmin, vmax + 1))
        r = math.exp(rng.uniform(math.log(rmin), math.log(rmax))) * (1 + rng.uniform(-0.15, 0.15, n))
        t = 2 * np.pi * np.arange(n) / n
        out.append(np.stack([c[0] + r * np.cos(t), c[1] + r * np.sin(t)], 1))
    return out


def _gon(n=256, r=0.45, c=0.5):
    t = 2 * np.pi * np.arange(n) / n
    return np.stack([c + r * np.cos(t), c + r * np.sin(t)], 1)


def _flat(case, seed):
    """[(centre, angle, loops, solid)] of the bodies of a 2-D case, positions [N, 2] and supports [N]."""
    n, h, g = case["n"], case["h"], _gen(seed)
    if case.get("shape") == "gon":
        bodies, lo, hi = [((0.0, 0.0), 0.0, [_gon()], "outside")], 0.05, 0.95
    elif case["what"] == "bodies":
        rng = np.random.default_rng(seed)
        tank = np.array([[0.0, 0.0], [4.0, 0.0], [4.0, 4.0], [0.0, 4.0]])
        edge = np.concatenate([a + (b - a) * np.arange(100)[:, None] / 100 for a, b in zip(tank, np.roll(tank, -1, 0))])
        bodies = [((0.0, 0.0), 0.0, [edge], "outside")]
        for _ in range(case["bodies"] - 1):
            star = _stars(int(rng.integers(1 << 31)), 1, 64, 256, box=0.0, rmin=0.1, rmax=0.4)
            bodies.append((tuple(float(v) for v in rng.uniform(0.6, 3.4, 2)), float(rng.uniform(-3, 3)), star, "inside"))
        lo, hi = 0.005, 3.995
    else:
        few = case["what"] == "adjoint"
        loops = _stars(seed, 16, 128, 128) if few else _stars(seed, STARS["stars"], STARS["vmin"], STARS["vmax"])
        posed = case["what"] == "delta"      # the delta+ body is turned and shifted
        bodies = [((0.3, -0.2) if posed else (0.0, 0.0), 0.4 if posed else 0.0, loops, "inside")]
        lo, hi = 0.0, 4.0
    pos = lo + (hi - lo) * torch.rand((n, 2), dtype=F64, device=DEV, generator=g)
    sup = torch.full((n,), h, dtype=F64, device=DEV)
    if case["what"] == "bodies":
        sup = h * (0.7 + 0.3 * torch.rand(n, dtype=F64, device=DEV, generator=g))
    return bodies, pos, sup


def _weights(case, seed):
    g = _gen(seed + 977)
    n = case["n"]
    return [torch.randn(s, dtype=F64, device=DEV, generator=g) for s in ((n,), (n, 2), (n, 2, 2))]


def _fibres(case, seed):
    """centres [M, 2] and radii [M] of non-overlapping disks in [0, 4]^2, radii 0.5 to 5 times 0.02."""
    rng = np.random.default_rng(seed)
    C, R = np.zeros((0, 2)), np.zeros(0)
    for _ in range(40 * case["disks"]):
        if len(R) == case["disks"]:
            break
        c, r = rng.uniform(0, 4, 2), rng.uniform(0.01, 0.1) * (1.0 if len(R) < 300 else 0.5)
        if not len(R) or (np.hypot(*(C - c).T) > R + r).all():
            C, R = np.concatenate([C, c[None]]), np.append(R, r)
    return C, R


def _icosphere(k, seed, radius=0.6, jitter=0.05):
    t = (1 + 5 ** 0.5) / 2
    V = np.array([(-1, t, 0), (1, t, 0), (-1, -t, 0), (1, -t, 0), (0, -1, t), (0, 1, t), (0, -1, -t), (0, 1, -t),
                  (t, 0, -1), (t, 0, 1), (-t, 0, -1), (-t, 0, 1)], float)
    Fc = np.array([(0, 11, 5), (0, 5, 1), (0, 1, 7), (0, 7, 10), (0, 10, 11), (1, 5, 9), (5, 11, 4), (11, 10, 2),
                   (10, 7, 6), (7, 1, 8), (3, 9, 4), (3, 4, 2), (3, 2, 6), (3, 6, 8), (3, 8, 9), (4, 9, 5), (2, 4, 11),
                   (6, 2, 10), (8, 6, 7), (9, 8, 1)])
    for _ in range(k):
        e = np.sort(np.concatenate([Fc[:, [0, 1]], Fc[:, [1, 2]], Fc[:, [2, 0]]]), axis=1)
        u, inv = np.unique(e, axis=0, return_inverse=True)
        ab, bc, ca = inv.reshape(3, -1) + len(V)
        V = np.concatenate([V, (V[u[:, 0]] + V[u[:, 1]]) / 2])
        a, b, c = Fc.T
        Fc = np.concatenate([np.stack(x, 1) for x in ((a, ab, ca), (b, bc, ab), (c, ca, bc), (ab, bc, ca))])
    V = radius * V / np.linalg.norm(V, axis=1, keepdims=True)
    V = V * (1 + jitter * np.random.default_rng(seed).uniform(-1, 1, (len(V), 1)))
    return V, Fc.astype(np.int32)


def _solid(case, seed):
    """vertices, faces, queries [N, 3] of a mesh case; `near`: within about a support of the surface."""
    V, Fc = _icosphere(case["subdivisions"], seed)
    g, n = _gen(seed), case["n"]
    if case["near"]:
        d = torch.randn((n, 3), dtype=F64, device=DEV, generator=g)
        r = 0.6 + 1.5 * case["h"] * (2 * torch.rand((n, 1), dtype=F64, device=DEV, generator=g) - 1)
        return V, Fc, r * d / d.norm(dim=1, keepdim=True)
    return V, Fc, 2 * torch.rand((n, 3), dtype=F64, device=DEV, generator=g) - 1


def _rows(case, seed):
    """distances, normals, radii (None for half-spaces) of the radial rows."""
    g, n, h = _gen(seed), case["n"], case["h"]
    d = h * (2.4 * torch.rand(n, dtype=F64, device=DEV, generator=g) - 1.2)
    nrm = torch.randn((n, 3), dtype=F64, device=DEV, generator=g)
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    if case["what"] == "planes":
        return d, nrm, None
    R = h * 0.2 * torch.exp(math.log(250.0) * torch.rand(n, dtype=F64, device=DEV, generator=g))
    return torch.maximum(d, -R), nrm, R


def prepare(case, seed):
    from warpsphboundaries_b200 import AnalyticBoundary, Body, KernelFunctions, ParticleState, Scene, SurfaceRep
    what = case["what"]
    if what in ("spheres", "planes"):
        from warpsphboundaries_b200.radial import RadialEvaluator
        d, nrm, R = _rows(case, seed)
        ev = RadialEvaluator("plane" if what == "planes" else "sphere", kernel=case["kernel"], device=DEV)
        return what, ev.prepare(d, nrm, case["h"], **({} if R is None else {"radii": R}))
    if what == "mesh":
        from warpsphboundaries_b200.mesh3d import Evaluator, Geometry
        V, Fc, Q = _solid(case, seed)
        return what, Evaluator(Geometry.closed_surface(V, Fc), kernel=case["kernel"], device=DEV).prepare(Q, case["h"])
    if what == "disks":
        from warpsphboundaries_b200.scene import DiskArrayRep
        C, R = _fibres(case, seed)
        pos = 4.0 * torch.rand((case["n"], 2), dtype=F64, device=DEV, generator=_gen(seed))
        sup = torch.full((case["n"],), case["h"], dtype=F64, device=DEV)
        bodies = [Body(reps=[DiskArrayRep(C, R)])]
    else:
        described, pos, sup = _flat(case, seed)
        bodies = [Body(bodyId=i, center=c, angle=a, reps=[SurfaceRep.loops(loops, solid=solid)])
                  for i, (c, a, loops, solid) in enumerate(described)]
    scene = Scene(bodies, DEV)
    ps = ParticleState(pos, sup)
    state = {"provider": AnalyticBoundary(scene), "scene": scene, "ps": ps, "h": case["h"]}
    if "kernel" in case:
        state["kernel"] = getattr(KernelFunctions, SCHEME[case["kernel"]])
    if what == "groups":
        from warpsphboundaries_b200.provider import FusedGroup
        state["groups"] = tuple(FusedGroup(k) for k in case["kernels"].split(","))
    if what == "adjoint":
        pos.requires_grad_(True)
        bodies[0].reps[0].vertices.requires_grad_(True)
        state["weights"] = _weights(case, seed)
    return what, state


# ------------------------------------------------------------------------------------------------------------ one pass
def run(state):
    what, s = state
    if what in ("spheres", "planes", "mesh"):
        return {"values": s.launch()}
    if what == "groups":
        from warpsphboundaries_b200.provider import FusedWall
        fw = FusedWall(s["scene"], s["ps"], s["h"], s["groups"])
        return [dict(r) for r in fw.res]
    if what == "adjoint":
        from warpsphboundaries_b200.autograd import aggregate_moments
        body = s["scene"].bodies[0]
        rep, pos = body.reps[0], s["ps"].positions
        out = aggregate_moments(body, rep, pos, s["ps"].supports, s["kernel"], s["h"])
        vals = [out["lam"], out["m1"], out["m2"]]
        dx, dv = torch.autograd.grad(vals, [pos, rep.vertices], s["weights"])
        return {"lam": vals[0].detach(), "m1": vals[1].detach(), "m2": vals[2].detach(), "dx": dx, "dv": dv}
    if what == "distance":
        d, n, hit = s["provider"].signed_distance(s["ps"].positions, supportMax=s["h"])
        return {"d": d, "n": n, "hit": hit}
    from warpsphboundaries_b200 import WallOutput
    lean = what != "delta"
    fw = s["provider"].aggregate(s["ps"], s["h"], kernel=s["kernel"], laplacian=not lean, lean=lean)
    return {**fw.out, **fw.evaluate((WallOutput("m1", 0, "m1"), WallOutput("m2", 0, "m2")))}


# ------------------------------------------------------------------------------------------------------------ the work
PAIR_FLOPS = {"cubic": 386, "w2": 246, "w4": 313, "w6": 380, "delta": 246 + 150 + 180 + 20 * 25}


def _pairs(case):
    """expected neighbour pairs of a 2-D case: every edge of length l is met from the area 2 h l + pi h^2 around it."""
    n, h = case["n"], case["h"]
    if case.get("shape") == "gon":
        edges, ell, area = 256, 2 * math.pi * 0.45 / 256, 0.81
    elif case["what"] == "bodies":
        edges, ell, area = 400 + 160 * (case["bodies"] - 1), 0.03, 16.0
    elif case["what"] == "adjoint":
        edges, ell, area = 16 * 128, 0.108 * 0.168, 16.0
    else:
        edges, ell, area = 64 * 272, 0.105 * 0.168, 16.0
    return n / area * edges * (2 * h * ell + math.pi * h * h)


def work(case):
    what, n = case["what"], case["n"]
    if what in ("spheres", "planes"):      # in: d, n, h (R); out: 28 channels; about 8 nodes of 60 operations a row
        return {"bytes": n * 8.0 * (5 + (what == "spheres") + 28), "flops": n * 500.0}
    if what == "mesh":
        h, faces = case["h"], 20 * 4 ** case["subdivisions"]
        area = 4 * math.pi * 0.36
        near = area * 2 * h                                    # the shell around the surface
        per_row = math.pi * h * h * 0.75 * faces / area + 6    # faces a near query meets
        rows = n * (2.0 / 3.0 if case["near"] else near / 8.0)
        return {"bytes": n * 8.0 * 32, "flops": rows * per_row * 2000.0}
    if what == "disks":
        arcs = 2 * math.pi * 0.04 * case["disks"] * 2 * case["h"] / 16.0   # particles within a support of a circle
        return {"bytes": n * 8.0 * 16, "flops": n * arcs * 24 * 60.0}
    if what == "distance":
        return {"bytes": n * 8.0 * 5, "flops": n * 300.0}
    pairs = _pairs(case)
    if what == "groups":
        ks = case["kernels"].split(",")
        return {"bytes": n * 8.0 * (3 + 13 * len(ks)), "flops": pairs * sum(PAIR_FLOPS[k] for k in ks)}
    if what == "adjoint":
        return {"bytes": n * 8.0 * (3 + 7 + 7 + 2), "flops": pairs * (PAIR_FLOPS[case["kernel"]] + 300.0)}
    if what == "delta":
        return {"bytes": n * 8.0 * (3 + 13 + 2 + 1 + 2), "flops": pairs * PAIR_FLOPS["delta"]}
    return {"bytes": n * 8.0 * (3 + 13 * case.get("bodies", 1)), "flops": pairs * PAIR_FLOPS[case["kernel"]]}


# ------------------------------------------------------------------------------------------------------------ exact values
def _pmul(a, b):
    out = [F(0)] * (len(a) + len(b) - 1)
    for i, x in enumerate(a):
        for j, y in enumerate(b):
            out[i + j] += x * y
    return out


def _ppow(a, k):
    out = [F(1)]
    for _ in range(k):
        out = _pmul(out, a)
    return out


def _shape(name):
    """blocks [(R, coefficients)] of the unnormalised kernel: sum of P(r) on r < R."""
    one = [F(1), F(-1)]
    if name == "cubic":
        return [(F(1), _ppow(one, 3)), (F(1, 2), [-4 * x for x in _ppow([F(1, 2), F(-1)], 3)])]
    if name == "cone":
        return [(F(1), one)]
    if name == "lw2":
        return [(F(1), _ppow(one, 3))]
    if name == "lw4":
        p, q = _ppow(one, 5), _ppow(one, 6)
        return [(F(1), [6 * (p[i] if i < len(p) else 0) - 5 * q[i] for i in range(len(q))])]
    n, poly = {"w2": (4, [F(1), F(4)]), "w4": (6, [F(1), F(6), F(35, 3)]), "w6": (8, [F(1), F(8), F(25), F(32)])}[name]
    return [(F(1), _pmul(_ppow(one, n), poly))]


def _normalised(name, dim):
    """the blocks with int W = 1 over the plane (dim 2) or space (dim 3); pi is divided out (W = blocks / pi)."""
    blocks = _shape(name)
    tot = sum(sum(c * R ** (k + dim) / (k + dim) for k, c in enumerate(P)) for R, P in blocks)
    scale = 1 / (2 * tot) if dim == 2 else 1 / (4 * tot)
    return [(R, [scale * c for c in P]) for R, P in blocks]


def _poly(c, x):
    v = torch.full_like(x, float(c[-1]))
    for a in reversed(c[:-1]):
        v = v * x + float(a)
    return v


def _panels(u0, u1, base):
    """(index, lo, hi) of the panels [0, 2 base], [2 base, 4 base], ... of every interval [u0, u1] (u0 >= 0)."""
    edge = torch.zeros_like(base)
    top = 2 * base
    for _ in range(80):
        lo, hi = torch.maximum(u0, edge), torch.minimum(u1, top)
        idx = torch.nonzero(hi > lo).flatten()
        if len(idx):
            yield idx, lo[idx], hi[idx]
        if not bool((u1 > top).any()):
            return
        edge, top = top, 2 * top


def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return torch.tensor(x, dtype=F64, device=DEV), torch.tensor(w, dtype=F64, device=DEV)


def _seg_pairs(X, sup, V, E):
    """(row, edge) of every segment closer than the row's support."""
    rows, es = [], []
    a, b = V[E[:, 0]], V[E[:, 1]]
    d = b - a
    dd = (d * d).sum(1)
    step = max(1, (1 << 26) // max(1, len(E)))
    for i in range(0, len(X), step):
        x = X[i:i + step]
        rx, ry = x[:, None, 0] - a[None, :, 0], x[:, None, 1] - a[None, :, 1]
        t = ((rx * d[:, 0] + ry * d[:, 1]) / dd).clamp(0, 1)
        q = (rx - t * d[:, 0]).square() + (ry - t * d[:, 1]).square()
        k = torch.nonzero(q < sup[i:i + step, None].square())
        rows.append(k[:, 0] + i)
        es.append(k[:, 1])
    return torch.cat(rows), torch.cat(es)


def _winding(X, V, E, background):
    out = torch.empty(len(X), dtype=F64, device=DEV)
    a, b = V[E[:, 0]], V[E[:, 1]]
    step = max(1, (1 << 26) // max(1, len(E)))
    for i in range(0, len(X), step):
        x = X[i:i + step]
        ax, ay = a[None, :, 0] - x[:, None, 0], a[None, :, 1] - x[:, None, 1]
        cx, cy = b[None, :, 0] - x[:, None, 0], b[None, :, 1] - x[:, None, 1]
        cr = ax * cy - ay * cx
        up = (ay <= 0) & (cy > 0) & (cr > 0)
        down = (cy <= 0) & (ay > 0) & (cr < 0)
        out[i:i + step] = up.sum(1).to(F64) - down.sum(1).to(F64)
    return out + background


class _Chords:
    """the pairs of one body: frames in units of the support, and integrals over the chords inside a radius."""

    def __init__(self, X, sup, V, E):
        self.rows, self.es = _seg_pairs(X, sup, V, E)
        self.h = sup[self.rows]
        p = (V[E[self.es, 0]] - X[self.rows]) / self.h[:, None]
        q = (V[E[self.es, 1]] - X[self.rows]) / self.h[:, None]
        d = q - p
        ell = d.norm(dim=1)
        self.t = d / ell[:, None]
        self.n = torch.stack([self.t[:, 1], -self.t[:, 0]], 1)
        self.z = (p[:, 0] * q[:, 1] - p[:, 1] * q[:, 0]) / ell
        self.s0, self.s1 = (self.t * p).sum(1), (self.t * q).sum(1)
        self.gx, self.gw = _gauss(24)

    def clip(self, R):
        L = (R * R - self.z * self.z).clamp(min=0).sqrt()
        lo, hi = torch.maximum(self.s0, -L), torch.minimum(self.s1, L)
        empty = (self.z.abs() >= R) | (hi <= lo)
        return torch.where(empty, torch.zeros_like(lo), lo), torch.where(empty, torch.zeros_like(hi), hi)

    def integrate(self, R, funcs):
        """[sum over the chord inside r < R of f(r, s)] for every f."""
        lo, hi = self.clip(R)
        out = [torch.zeros_like(self.z) for _ in funcs]
        base = self.z.abs().clamp(min=2.0 ** -30)
        for sgn, u0, u1 in ((-1.0, (-hi).clamp(min=0), -lo), (1.0, lo.clamp(min=0), hi)):
            for idx, a, b in _panels(u0, u1, base):
                for k in range(0, len(idx), 1 << 20):
                    i = idx[k:k + (1 << 20)]
                    hc, mc = 0.5 * (b - a)[k:k + (1 << 20)], 0.5 * (b + a)[k:k + (1 << 20)]
                    u = hc[:, None] * self.gx + mc[:, None]
                    r = (u * u + self.z[i, None].square()).sqrt()
                    for f, o in zip(funcs, out):
                        o[i] += hc * (f(r, sgn * u) * self.gw).sum(1)
        return out

    def angle(self, R):
        lo, hi = self.clip(R)
        z = self.z
        return torch.where(hi > lo, torch.atan2(z * (hi - lo), z * z + lo * hi), torch.zeros_like(z))


def _scatter(n, rows, v):
    out = torch.zeros((n,) + tuple(v.shape[1:]), dtype=F64, device=DEV)
    return out.index_add_(0, rows, v)


def _wall_exact(ch, ind, sup, name, n):
    """lam, G, Cov, m1, m2 of one body for one kernel (frames of `ch` are in the world frame)."""
    z, nx, t = ch.z, ch.n, ch.t
    lam, psi2 = torch.zeros_like(z), torch.zeros_like(z)
    W0, W1, P0, P1 = (torch.zeros_like(z) for _ in range(4))
    mass = plane2 = 0.0
    for R, c in _normalised(name, 2):
        Rf = float(R)
        f1 = [x / (k + 2) for k, x in enumerate(c)]                       # F1(r) / r^2, F1 = int_0^r t P
        F1R = sum(x * R ** (k + 2) for k, x in enumerate(f1))
        psi = [-F1R, F(0)] + f1                                           # int t P from R
        f2 = [x / (k + 2) for k, x in enumerate(psi)]
        F2R = sum(x * R ** (k + 2) for k, x in enumerate(f2))
        a, b, c0, c1, p0, p1 = ch.integrate(Rf, [
            lambda r, s: _poly(f1, r), lambda r, s: _poly(f2, r), lambda r, s: _poly(c, r),
            lambda r, s: s * _poly(c, r), lambda r, s: _poly(psi, r), lambda r, s: s * _poly(psi, r)])
        ang = ch.angle(Rf)
        lam += z * a - float(F1R) * ang
        psi2 += z * b - float(F2R) * ang
        W0 += c0
        W1 += c1
        P0 += p0
        P1 += p1
        mass += 2 * float(F1R)
        plane2 -= 2 * float(F2R)
    pi = math.pi
    h, rows, eye = ch.h, ch.rows, torch.eye(2, dtype=F64, device=DEV)
    L = _scatter(n, rows, lam / pi) + ind * mass
    yW = nx * (z * W0)[:, None] + t * W1[:, None]
    yP = nx * (z * P0)[:, None] + t * P1[:, None]
    G = _scatter(n, rows, -nx * (W0 / pi / h)[:, None])
    cov = L[:, None, None] * eye - _scatter(n, rows, yW[:, :, None] * nx[:, None, :] / pi)
    m1 = _scatter(n, rows, nx * (P0 * h / pi)[:, None])
    m2 = _scatter(n, rows, (0.5 * (yP[:, :, None] * nx[:, None, :] + yP[:, None, :] * nx[:, :, None])
                            - psi2[:, None, None] * eye) * (h * h / pi)[:, None, None])
    m2 = m2 + (ind * plane2 * sup * sup)[:, None, None] * eye
    return {"lam": L, "G": G, "Cov": cov, "m1": m1, "m2": m2}


def _world(centre, angle, loops, solid):
    """world vertices and edges of a body, solid on the left."""
    V, E, off = [], [], 0
    for P in loops:
        area = (P[:, 0] * np.roll(P[:, 1], -1) - np.roll(P[:, 0], -1) * P[:, 1]).sum()
        P = P if (area > 0) == (solid == "inside") else P[::-1]
        k = np.arange(len(P))
        V.append(P)
        E.append(np.stack([off + k, off + (k + 1) % len(P)], 1))
        off += len(P)
    V = np.concatenate(V)
    c, s = math.cos(angle), math.sin(angle)
    V = V @ np.array([[c, s], [-s, c]]) + np.array(centre)
    return torch.tensor(V, dtype=F64, device=DEV), torch.tensor(np.concatenate(E), device=DEV)


def _flat_exact(case, seed):
    bodies, X, sup = _flat(case, seed)
    n, what = len(X), case["what"]
    names = case["kernels"].split(",") if what == "groups" else [case["kernel"]]
    extra = {"delta": ["cone", "l" + case.get("kernel", "")]}.get(what, [])
    per = []
    for centre, angle, loops, solid in bodies:
        V, E = _world(centre, angle, loops, solid)
        ch, ind = _Chords(X, sup, V, E), _winding(X, V, E, 1.0 if solid == "outside" else 0.0)
        got = [_wall_exact(ch, ind, sup, k, n) for k in names + extra]
        if what == "delta":
            power = {"w2": (4, [F(1), F(4)]), "w4": (6, [F(1), F(6), F(35, 3)])}[case["kernel"]]
            full = _pmul(_ppow([F(1), F(-1)], 5 * power[0]), _ppow(power[1], 5))
            C = float(1 / (2 * sum(c / (k + 2) for k, c in enumerate(full))))
            (w5,) = ch.integrate(1.0, [lambda r, s: C * ((1 - r) ** power[0] * _poly(power[1], r)) ** 5])
            got.append({"G": _scatter(n, ch.rows, -ch.n * (w5 / math.pi / ch.h)[:, None])})
        per.append(got)
    stack = lambda g, k: torch.stack([b[g][k] for b in per])  # noqa: E731
    out = [{k: stack(g, k) for k in ("lam", "G", "Cov", "m1", "m2")} for g in range(len(names))]
    if what == "groups":
        return out
    out = out[0]
    if what == "delta":
        lw = {k: stack(2, k) for k in ("lam", "Cov")}
        out.update(cover=stack(1, "G"), lap=2 * lw["lam"] - lw["Cov"][..., 0, 0] - lw["Cov"][..., 1, 1], tens=stack(3, "G"))
    return out


def _adjoint_exact(case, seed):
    bodies, X, sup = _flat(case, seed)
    (centre, angle, loops, solid), = bodies
    V, E = _world(centre, angle, loops, solid)
    n, ch = len(X), _Chords(X, sup, V, E)
    out = _wall_exact(ch, _winding(X, V, E, 0.0), sup, case["kernel"], n)
    wl, w1, w2 = _weights(case, seed)
    r, h, z = ch.rows, ch.h, ch.z
    # the weighted boundary integrand sum_alpha u_alpha y^alpha along the edge, y = z n + s t
    yn = z[:, None] * ch.n
    q = 0.5 * (w2[r] + w2[r].transpose(1, 2)) * h[:, None, None]
    bil = lambda a, b: torch.einsum("pi,pij,pj->p", a, q, b)  # noqa: E731
    f = [wl[r] / h + (w1[r] * yn).sum(1) + bil(yn, yn), (w1[r] * ch.t).sum(1) + 2 * bil(yn, ch.t), bil(ch.t, ch.t)]
    I = [torch.zeros_like(z) for _ in range(4)]
    for R, c in _normalised(case["kernel"], 2):
        got = ch.integrate(float(R), [lambda rr, s, k=k: s ** k * _poly(c, rr) for k in range(4)])
        I = [a + b for a, b in zip(I, got)]
    i0 = sum(fk * I[k] for k, fk in enumerate(f))
    i1 = sum(fk * I[k + 1] for k, fk in enumerate(f))
    a1 = (i1 - ch.s0 * i0) / (ch.s1 - ch.s0)
    dv = torch.zeros_like(V)
    dv.index_add_(0, E[ch.es, 0], ch.n * ((i0 - a1) / math.pi)[:, None])
    dv.index_add_(0, E[ch.es, 1], ch.n * (a1 / math.pi)[:, None])
    return {"lam": out["lam"], "m1": out["m1"], "m2": out["m2"], "dx": _scatter(n, r, -ch.n * (i0 / math.pi)[:, None]), "dv": dv}


def _distance_exact(case, seed):
    bodies, X, _ = _flat(case, seed)
    best = torch.full((len(X),), math.inf, dtype=F64, device=DEV)
    for centre, angle, loops, solid in bodies:
        V, E = _world(centre, angle, loops, solid)
        a, b = V[E[:, 0]], V[E[:, 1]]
        d = b - a
        dd = (d * d).sum(1)
        ins = _winding(X, V, E, 1.0 if solid == "outside" else 0.0) > 0.5
        step = max(1, (1 << 26) // len(E))
        for i in range(0, len(X), step):
            x = X[i:i + step]
            rx, ry = x[:, None, 0] - a[None, :, 0], x[:, None, 1] - a[None, :, 1]
            t = ((rx * d[:, 0] + ry * d[:, 1]) / dd).clamp(0, 1)
            q = ((rx - t * d[:, 0]).square() + (ry - t * d[:, 1]).square()).amin(1).sqrt()
            best[i:i + step] = torch.minimum(best[i:i + step], torch.where(ins[i:i + step], -q, q))
    return {"d": best, "n": None, "hit": None}     # the normal at a corner is a choice among the edges that meet there


def _disks_exact(case, seed):
    """per (particle, disk): the integrals over the radius r of W times the arc of the circle r inside the disk."""
    C, R = (torch.tensor(v, dtype=F64, device=DEV) for v in _fibres(case, seed))
    n, h = case["n"], case["h"]
    X = 4.0 * torch.rand((n, 2), dtype=F64, device=DEV, generator=_gen(seed))
    rows, ds = [], []
    step = (1 << 27) // max(1, len(R))
    for i in range(0, n, step):
        d2 = (X[i:i + step, None, 0] - C[None, :, 0]).square() + (X[i:i + step, None, 1] - C[None, :, 1]).square()
        k = torch.nonzero(d2 < (R + h).square())
        rows.append(k[:, 0] + i)
        ds.append(k[:, 1])
    rows, ds = torch.cat(rows), torch.cat(ds)
    v = (C[ds] - X[rows]) / h
    D, Rr = v.norm(dim=1).clamp(min=1e-300), R[ds] / h
    e = v / D[:, None]
    blocks = _normalised(case["kernel"], 2)
    S = torch.zeros((6, len(D)), dtype=F64, device=DEV)     # lam, m1, G, m2 iso, m2 aniso, (W' r iso, aniso below)
    T = torch.zeros((2, len(D)), dtype=F64, device=DEV)
    gx, gw = _gauss(24)

    def add(i, r, w, beta, sb, cb):
        """r, beta [p, k], weights w of dr: arcs |phi| < beta of the circles r."""
        for Rb, c in blocks:
            inb = (r < float(Rb)).to(F64) * w
            dc = [k * x for k, x in enumerate(c)][1:] or [F(0)]
            W, dW = _poly(c, r) * inb, _poly(dc, r) * inb
            iso, ani = beta, sb * cb
            S[0, i] += (2 * W * r * beta).sum(1)
            S[1, i] += (2 * W * r * r * sb).sum(1)
            S[2, i] -= (2 * dW * r * sb).sum(1)
            S[3, i] += (W * r ** 3 * iso).sum(1)
            S[4, i] += (W * r ** 3 * ani).sum(1)
            T[0, i] -= (dW * r * r * iso).sum(1)
            T[1, i] -= (dW * r * r * ani).sum(1)

    knots = sorted({0.0, 1.0, *(float(Rb) for Rb, _ in blocks)})
    for k0, k1 in zip(knots[:-1], knots[1:]):
        full = (Rr - D).clamp(min=k0, max=k1)                    # circles wholly inside the disk
        i = torch.nonzero(full > k0).flatten()
        for k in range(0, len(i), 1 << 20):
            j = i[k:k + (1 << 20)]
            hc, mc = 0.5 * (full[j] - k0), 0.5 * (full[j] + k0)
            r = hc[:, None] * gx + mc[:, None]
            add(j, r, hc[:, None] * gw, torch.full_like(r, math.pi), torch.zeros_like(r), torch.ones_like(r))
        dm = (D - Rr).abs()
        lo, hi = dm.clamp(min=k0), (D + Rr).clamp(max=k1)
        # panels graded from |D - R|, mapped by a cosine so that the square roots at both ends are smooth
        for j, a, b in _panels((lo - dm).clamp(min=0), hi - dm, (0.5 * dm).clamp(min=2.0 ** -40)):
            for k in range(0, len(j), 1 << 19):
                i = j[k:k + (1 << 19)]
                a_, b_ = a[k:k + (1 << 19), None], b[k:k + (1 << 19), None]
                th = 0.5 * math.pi * (gx + 1)
                x = a_ + (b_ - a_) * torch.sin(0.5 * th).square()      # r - |D - R|
                w = 0.25 * math.pi * (b_ - a_) * torch.sin(th) * gw
                Di, Ri, mi = D[i, None], Rr[i, None], dm[i, None]
                r = mi + x
                # sin^2(beta / 2) = (R^2 - (D - r)^2) / (4 r D), each factor without cancellation at its end
                near = torch.where(Di >= Ri, x, 2 * mi + x)           # R - D + r
                far = torch.where(Di >= Ri, 2 * Ri - x, 2 * Di - x)   # R + D - r
                s2 = (near * far / (4 * r * Di)).clamp(0, 1)
                beta = 2 * torch.asin(s2.sqrt())
                add(i, r, w, beta, torch.sin(beta), torch.cos(beta))
    eye = torch.eye(2, dtype=F64, device=DEV)
    ee = e[:, :, None] * e[:, None, :]
    tensor = lambda iso, ani: iso[:, None, None] * eye + ani[:, None, None] * (2 * ee - eye)  # noqa: E731
    pi = math.pi
    out = {"lam": _scatter(n, rows, S[0] / pi), "G": _scatter(n, rows, e * (S[2] / pi / h)[:, None]),
           "Cov": _scatter(n, rows, tensor(T[0], T[1]) / pi), "m1": _scatter(n, rows, e * (S[1] * h / pi)[:, None]),
           "m2": _scatter(n, rows, tensor(S[3], S[4]) * (h * h / pi))}
    return {k: v[None] for k, v in out.items()}


def _baseline(lam, m1, m2, G, g1, H):
    """[N, 28]: value moments, gradient moments, Hessian."""
    n = len(lam)
    up = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]
    sym = lambda m: torch.stack([m[:, i, j] for i, j in up], 1)  # noqa: E731
    return torch.cat([lam[:, None], m1, sym(m2), G, g1.reshape(n, 9), sym(H)], 1)


def _radial_exact(case, seed):
    """per row: integrals over the radius of the cap the sphere r cuts from the solid (axis = outward normal)."""
    d, nrm, R = _rows(case, seed)
    n, h = case["n"], case["h"]
    d = d / h
    rad = None if R is None else R / h
    v = torch.zeros((9, n), dtype=F64, device=DEV)
    gx, gw = _gauss(24)
    end = torch.ones_like(d) if rad is None else (2 * rad + d).clamp(max=1.0)
    for Rb, c in _normalised(case["kernel"], 3):
        Rb = float(Rb)
        dc = [k * x for k, x in enumerate(c)][1:]                        # W'
        ddc = [k * x for k, x in enumerate(dc)][1:] or [F(0)]            # W''
        for lo, hi, cap in ((torch.zeros_like(d), (-d).clamp(0, Rb), False), (d.abs(), end.clamp(max=Rb), True)):
            idx = torch.nonzero(hi > lo).flatten()
            for k in range(0, len(idx), 1 << 19):
                i = idx[k:k + (1 << 19)]
                hc, mc = 0.5 * (hi - lo)[i], 0.5 * (hi + lo)[i]
                r = hc[:, None] * gx + mc[:, None]
                w = hc[:, None] * gw
                if cap:
                    di = d[i, None]
                    if rad is None:
                        u, vv = (r - di) / r, (r + di) / r
                    else:
                        Ri = rad[i, None]
                        two = 2 * (Ri + di) * r
                        u, vv = (r - di) * (2 * Ri + di - r) / two, (r + di) * (2 * Ri + di + r) / two
                else:
                    u, vv = torch.full_like(r, 2.0), torch.zeros_like(r)
                cp = 0.5 * (u - vv)
                a0, a1, at, an = 2 * u, -u * vv, u * u * (1 + vv) / 3, 2 / 3 * u * (cp * cp - cp + 1)
                W, dW, ddW = _poly(c, r), _poly(dc, r), _poly(ddc, r)
                for q, f in enumerate((W * r ** 2 * a0, W * r ** 3 * a1, W * r ** 4 * at, W * r ** 4 * an,
                                       -dW * r ** 2 * a1, -dW * r ** 3 * at, -dW * r ** 3 * an,
                                       r * dW * a0 + (ddW * r ** 2 - dW * r) * at, r * dW * a0 + (ddW * r ** 2 - dW * r) * an)):
                    v[q, i] += (w * f).sum(1)
    eye = torch.eye(3, dtype=F64, device=DEV)
    nn = nrm[:, :, None] * nrm[:, None, :]
    ten = lambda t, a: t[:, None, None] * eye + (a - t)[:, None, None] * nn  # noqa: E731
    return {"values": _baseline(v[0], nrm * (v[1] * h)[:, None], ten(v[2], v[3]) * h * h, nrm * (v[4] / h)[:, None],
                                ten(v[5], v[6]), ten(v[7], v[8]) / h ** 2)}


class _Laurent:
    """a piecewise Laurent polynomial on [0, 1] with exact coefficients: pieces [(lo, hi, {power: coefficient})]."""

    def __init__(self, pieces):
        self.pieces = pieces

    @staticmethod
    def at(d, x):
        return sum((c * x ** e for e, c in d.items()), F(0))

    def potential(self):
        """A with A' = r f and A(1) = 0."""
        out, tail = [], F(0)
        for lo, hi, d in reversed(self.pieces):
            A = {e + 2: c / (e + 2) for e, c in d.items() if c}
            A[0] = A.get(0, F(0)) + tail - self.at(A, hi)
            tail = self.at(A, lo) if lo > 0 else F(0)
            out.append((lo, hi, A))
        return _Laurent(out[::-1])

    def __call__(self, r, z=None, power=0):
        """z^power f(r), 0 beyond r = 1; negative powers of r are met by the powers of z first."""
        out = torch.zeros_like(r)
        for lo, hi, d in self.pieces:
            inside = (r >= float(lo)) & (r < float(hi))
            top, low = max(d), min(min(d), 0)
            v = _poly([d.get(e, F(0)) for e in range(0, top + 1)], r)
            v = v * z ** power if power else v
            for e in range(low, 0):
                if d.get(e):
                    v = v + float(d[e]) * (z / r) ** (-e) * z ** (power + e)
            out = torch.where(inside, v, out)
        return out


def _solid_tables(name):
    blocks = sorted(_normalised(name, 3), key=lambda b: b[0])
    pieces, lo = [], F(0)
    for R, _ in blocks:
        c = {}
        for R2, P in blocks:
            if R2 >= R:
                for k, x in enumerate(P):
                    c[k] = c.get(k, F(0)) + x
        pieces.append((lo, R, c))
        lo = R
    K, Q1 = [], []
    for k in range(3):
        acc, qs = F(0), []
        for lo, hi, c in pieces:
            q = {e + 3 + k: x / (e + 3 + k) for e, x in c.items()}
            q[0] = acc - _Laurent.at(q, lo)
            acc = _Laurent.at(q, hi)
            qs.append((lo, hi, q))
        Q1.append(acc)
        for i, (lo, hi, q) in enumerate(qs):
            q[0] -= acc
            qs[i] = (lo, hi, {e - 3 - k: x for e, x in q.items() if x})
        K.append(_Laurent(qs))
    W = _Laurent(pieces)
    L = _Laurent([(lo, hi, {e - 2: e * x for e, x in c.items() if e}) for lo, hi, c in pieces])
    A = [K[0].potential(), K[1].potential(), K[2].potential(), W.potential(), L.potential()]
    return A + [A[2].potential()], [float(q) for q in Q1], float(pieces[0][1])


def _mesh_exact(case, seed):
    V, Fc, Q = _solid(case, seed)
    V, Fc = torch.tensor(V, dtype=F64, device=DEV), torch.tensor(Fc, dtype=torch.long, device=DEV)
    h, n = case["h"], len(Q)
    P = V[Fc]                                                            # [faces, 3, 3]
    cen = P.mean(1)
    reach = (P - cen[:, None]).norm(dim=2).amax(1) + h
    N = torch.linalg.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0])
    N = N / N.norm(dim=1, keepdim=True)
    # the surface is star-shaped about the origin: only queries between its smallest and largest radius need the sum of
    # solid angles
    inner = (P * N[:, None]).sum(2).amin()
    rq = Q.norm(dim=1)
    ind = (rq < inner).to(F64)
    unsure = torch.nonzero((rq >= inner) & (rq <= V.norm(dim=1).max())).flatten()
    step = max(1, (1 << 25) // len(Fc))
    for k in range(0, len(unsure), step):
        i = unsure[k:k + step]
        a, b, c = (P[None, :, j] - Q[i, None] for j in range(3))
        la, lb, lc = a.norm(dim=2), b.norm(dim=2), c.norm(dim=2)
        det = (a * torch.linalg.cross(b, c)).sum(2)
        den = la * lb * lc + (a * b).sum(2) * lc + (b * c).sum(2) * la + (c * a).sum(2) * lb
        ind[i] = torch.round(2 * torch.atan2(det, den).sum(1) / (4 * math.pi))
    out = torch.zeros((n, 28), dtype=F64, device=DEV)
    A, Q1, knot = _solid_tables(case["kernel"])
    eye = torch.eye(3, dtype=F64, device=DEV)
    near = torch.nonzero((rq > inner - h) & (rq < V.norm(dim=1).max() + h)).flatten()
    gx, gw = _gauss(16)
    powers = (1, 2, 3, 0, 0, 1)
    step = max(1, (1 << 27) // len(Fc))
    for k in range(0, len(near), step):
        i = near[k:k + step]
        d2 = (Q[i].square().sum(1)[:, None] + cen.square().sum(1)[None] - 2 * Q[i] @ cen.T)
        pr = torch.nonzero(d2 < (reach * (1 + 1e-9)).square()[None])
        for m in range(0, len(pr), 1 << 17):
            rows, f = i[pr[m:m + (1 << 17), 0]], pr[m:m + (1 << 17), 1]
            Nf = N[f]
            p = (P[f] - Q[rows][:, None]) / h                            # [pairs, 3, 3]
            q = p.roll(-1, 1)
            ell = (q - p).norm(dim=2)
            t = (q - p) / ell[..., None]
            mu = torch.linalg.cross(t, Nf[:, None].expand_as(t))
            z1 = (p[:, 0] * Nf).sum(1)
            z1 = torch.where(z1.abs() < 1e-60, torch.full_like(z1, 1e-60), z1)
            w, s0 = (mu * p).sum(2).reshape(-1), (t * p).sum(2).reshape(-1)
            s1 = s0 + ell.reshape(-1)
            z = z1[:, None].expand(-1, 3).reshape(-1)
            c2 = z * z + w * w
            c = c2.sqrt()
            Lc = (1 - c2).clamp(min=0).sqrt()
            lo, hi = torch.maximum(s0, -Lc), torch.minimum(s1, Lc)
            none = (c2 >= 1) | (hi <= lo)
            lo, hi = torch.where(none, torch.zeros_like(lo), lo), torch.where(none, torch.zeros_like(hi), hi)
            Aa = [a(z.abs(), z, e) for a, e in zip(A, powers)]
            S = torch.zeros((12, len(z)), dtype=F64, device=DEV)         # J of the six, then the six line integrals
            kn = (knot * knot - c2).clamp(min=0).sqrt() if knot < 1 else torch.zeros_like(c)
            for sgn, u0, u1 in ((-1.0, (-hi).clamp(min=0), -lo), (1.0, lo.clamp(min=0), hi)):
                for v0, v1 in ((u0, torch.minimum(u1, kn)), (torch.maximum(u0, kn), u1)):
                    for idx, a, b in _panels(v0, v1, (0.5 * c).clamp(min=2.0 ** -30)):
                        hc, mc = 0.5 * (b - a), 0.5 * (b + a)
                        u = hc[:, None] * gx + mc[:, None]
                        r = (u * u + c2[idx, None]).sqrt()
                        zi, wt = z[idx, None], hc[:, None] * gw
                        over = wt * w[idx, None] / (u * u + (w * w)[idx, None]).clamp(min=1e-300)
                        vals = [f_(r, zi, e) for f_, e in zip(A, powers)]
                        for j in range(6):
                            S[j, idx] += ((vals[j] - Aa[j][idx, None]) * over).sum(1)
                        k2 = A[2](r, zi, 3) / zi
                        S[6, idx] += (wt * vals[1]).sum(1) / z[idx]       # z int A_K1
                        S[7, idx] += (wt * k2).sum(1)                     # z^2 int A_K2
                        S[8, idx] += (wt * k2 / zi).sum(1)                # z int A_K2
                        S[9, idx] += (wt * sgn * u * k2 / zi).sum(1)      # z int s A_K2
                        S[10, idx] += (wt * vals[3]).sum(1)
                        S[11, idx] += (wt * vals[4]).sum(1)
            ang = lambda x0, x1: torch.where(x1 > x0, torch.atan2(w * (x1 - x0), w * w + x0 * x1), torch.zeros_like(w))  # noqa: E731,B023
            beyond = torch.where(none, ang(s0, s1), ang(s0, lo) + ang(hi, s1))
            for j in range(6):
                S[j] -= Aa[j] * beyond
            S = S.reshape(12, -1, 3)
            J = S[:6].sum(2)
            e = lambda a: torch.einsum("pe,pei->pi", a, mu)  # noqa: E731,B023
            w3 = w.reshape(-1, 3)
            NN = Nf[:, :, None] * Nf[:, None, :]
            both = lambda a: Nf[:, :, None] * a[:, None, :] + a[:, :, None] * Nf[:, None, :]  # noqa: E731,B023
            mt = torch.einsum("pe,pei,pej->pij", S[9], mu, t)
            m2 = (NN * (J[2] + J[5])[:, None, None] + both(e(S[7])) + torch.einsum("pe,pei,pej->pij", S[8] * w3, mu, mu)
                  + 0.5 * (mt + mt.transpose(1, 2)) - J[5][:, None, None] * eye)
            H = NN * (z1 * J[4])[:, None, None] + 0.5 * both(e(S[11]))
            g1 = -NN * (z1 * J[3])[:, None, None] - e(S[10])[:, :, None] * Nf[:, None, :]
            m1 = Nf * J[1][:, None] + e(S[6])
            out.index_add_(0, rows, _baseline(J[0], m1 * h, m2 * h * h, -Nf * (J[3] / h)[:, None], g1, H / h ** 2) / math.pi)
    out[:, 0] += ind * 4 * Q1[0]
    for c in (4, 7, 9):
        out[:, c] += ind * 4 / 3 * Q1[2] * h * h
    for c in (13, 17, 21):
        out[:, c] += out[:, 0]
    return {"values": out}


def exact(case, seed):
    what = case["what"]
    with torch.no_grad():
        if what in ("spheres", "planes"):
            return _radial_exact(case, seed)
        if what == "mesh":
            return _mesh_exact(case, seed)
        if what == "disks":
            return _disks_exact(case, seed)
        if what == "adjoint":
            return _adjoint_exact(case, seed)
        if what == "distance":
            return _distance_exact(case, seed)
        return _flat_exact(case, seed)
