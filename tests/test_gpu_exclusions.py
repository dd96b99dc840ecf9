"""The Ewald exclusion terms of the mixed path, -erf(alpha r)/r between the sites
of a molecule: lone waters against the FP64 path, over alpha r from 0.02 to 3 (a
series below 0.7, the error function above), with kept lists too."""
import numpy as np
import pytest

import macsimus_gb300 as M
from macsimus_gb300 import configs

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


@pytest.mark.parametrize("alpha", [0.02, 0.1, 0.29, 0.43, 0.5, 0.7, 1.0, 1.9])
@pytest.mark.parametrize("kw", [{}, dict(skin=1.0)], ids=["cells", "list"])
def test_exclusions_of_lone_waters(alpha, kw):
    L = 40.0
    system, r, _ = configs.build(["WAT"], [4], L, seed=4)   # 28 A apart
    ew = ([L] * 3, 10.0, alpha, 1.01 / L)
    # without the k-space part
    def forces(**k):
        fp = M.ForcePath(system, *ew, **k)
        return fp.forces(r)[0] - fp.ewald(r)[0]
    f64 = forces(precision="fp64")
    f = forces(kspace_engine=1, **kw)
    t = (alpha * 1.633) ** 2
    # eight roundings of the series; beyond it erf and exp to an ulp or two each,
    # the difference of the two 3 / (2 t) of its terms at t >= 1/2
    assert rel(f, f64) < (8 if t < 0.5 else 16) * 2.0 ** -24 * 2
    e64 = M.ForcePath(system, *ew, precision="fp64").forces(r, measure=True)[1]
    e = M.ForcePath(system, *ew, kspace_engine=1, **kw).forces(r, measure=True)[1]
    assert abs(e["er"] - e64["er"]) < 4e-7 * abs(e64["er"])
