"""The rounding of the closed-surface integrals against the reference's 30-digit values.

The potentials A_f are polynomials in r - R/2 (coefficients b_n).  A term of the face sums is b_n times an integral of
|t|^n, t up to R/2, or of the face's divided difference, whose terms reach (a + R/2)^n at a distance a of the query from the
face's plane; each carries a rounding of 2^-53 of itself.  The rows' faces lie at all distances below a support with most of
the kernel's weight near a = 0.3, so the root mean square error over the rows, in units of the support, is bounded by
2^-53 sum_blocks max_f sum_n |b_n| max(R/2, 0.3 R + R/2)^n.  (In powers of r the sums are 20 to 100 times larger.)"""
import json
from fractions import Fraction as F
from pathlib import Path

import numpy as np
import pytest
import torch

from warpsphboundaries_b200 import kernels as K
from warpsphboundaries_b200.mesh3d import ClosedMesh

pytestmark = pytest.mark.gpu
G = json.loads((Path(__file__).parent / "golden" / "mesh3d_golden.json").read_text())
DEV = torch.device("cuda")


def _bound(kernel):
    total = F(0)
    for t in K.mesh_blocks(kernel):
        R = F(t["R"])
        top = max(max(f) for f in t["funcs"].values())
        total += max(sum(abs(c) * (F(3, 10) * R + R / 2) ** n for n, c in enumerate(K.mesh_shifted(f, R / 2, top)))
                     for f in t["funcs"].values())
    return float(total) * 2.0 ** -53


@pytest.mark.parametrize("kernel", ["cubic", "w2", "w4", "w6"])
def test_rms_error_of_the_reference_rows(kernel):
    unit = np.concatenate([[0], np.full(3, -1), np.full(6, -2), np.full(3, 1), np.zeros(9), np.full(6, 2)])
    err = []
    for c in G["cases"]:
        if c["kernel"] != kernel:
            continue
        m, h = G["meshes"][c["mesh"]], c["h"]
        mesh = ClosedMesh(np.array(m["vertices"], float), np.array(m["faces"]), h, DEV)
        got = mesh.channels(torch.tensor([c["query"]], dtype=torch.float64, device=DEV),
                            torch.tensor([h], dtype=torch.float64, device=DEV), kernel).cpu().numpy()[0]
        err.append(np.abs((got - np.array([float(v) for v in c["values"]])) * h ** unit).max())
    assert len(err) == 17
    rms = float(np.sqrt(np.mean(np.square(err))))
    assert rms <= _bound(kernel), (rms, _bound(kernel))
