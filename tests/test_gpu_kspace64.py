"""The FP64 k-space sums and the adjoint's against the oracle: k sets of one
shell and of rows longer than a task's run, boxes with unequal edges, charge
counts around a CTA's 8 to 32, Drude charges; with and without a force loss."""
import numpy as np
import pytest

import macsimus_gb300 as M
from macsimus_gb300 import configs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("species,counts,L,kn", [
    (["NA", "CL"], [2, 1], [22.0, 22.0, 22.0], 1),       # 3 charges, six k vectors
    (["WAT"], [11], [20.0, 24.0, 21.0], 5),              # 33 charges
    (["WAT", "NA", "CL"], [30, 3, 2], [20.0, 20.0, 47.0], 9),   # |kz| to 21
    (["WATD"], [17], [19.0, 22.0, 20.0], 4),
    (["WAT"], [1700], [38.0, 37.0, 39.0], 8),            # 5100 charges: 16 a CTA
])
def test_matches_oracle(species, counts, L, kn):
    system, r, _ = configs.build(species, counts, min(L), seed=6)
    if system.polar:
        d = np.random.default_rng(1).normal(scale=0.05, size=r.shape)
        d[system.qpol == 0] = 0
        r = np.vstack([r, d])
    else:
        r = r + np.random.default_rng(2).normal(scale=0.1, size=r.shape)
    ew = (L, 9.2, 0.34, (kn + 1e-6) / min(L))
    fp = M.ForcePath(system, *ew, precision="fp64")
    f, e = fp.forces(r, measure=True)
    orc = O.Oracle(system, *ew)
    fo, eo = orc.forces(r, measure=True, nthreads=4)
    # the bounds of the FP64 path elsewhere
    assert np.sqrt(((f - fo) ** 2).sum() / (fo ** 2).sum()) < 1e-10
    assert abs(e["ek"] - eo["ek"]) <= 1e-10 * abs(eo["eself"])
    for m in range(6):
        assert abs(e["Pvir"][m] - eo["Pvir"][m]) <= 1e-9 * np.abs(eo["Pvir"]).max()
    if system.polar or system.ns > 1000:
        return
    g = np.random.default_rng(3).normal(size=f.shape) * 1e-3
    for gl in (g, None):
        a, o = fp.adjoint(r, gl), orc.adjoint(r, gl)
        assert abs(a["E"] - o["E"]) < 1e-10 * abs(eo["eself"])
        for k in ("dEp", "dWp", "dEq") + (("dLp", "dLq") if gl is not None else ()):
            assert np.abs(a[k] - o[k]).max() <= 1e-9 * np.abs(o[k]).max(), k
