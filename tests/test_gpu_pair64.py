"""The FP64 pair kernel (a warp per site, neighbours queued by class) against
the oracle: site counts around its sites per CTA, grids of one cell and of
many, a cutoff just short of half the box, kinds without Lennard-Jones term,
without charge and with neither, Drude shells; measured and plain forces."""
import numpy as np
import pytest

import macsimus_gb300 as M
from macsimus_gb300 import configs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("species,counts,L,cutoff", [
    (["WAT"], [11], 22.0, 10.9),                     # 33 sites, one cell
    (["WAT"], [216], 18.7, 9.3499),                  # the cutoff at half the box
    (["WAT", "NA", "CL", "PRB"], [300, 5, 5, 7], 28.0, 9.0),
    (["T4P", "PRB"], [170, 3], 20.0, 9.0),
    (["WATD"], [65], 20.0, 9.0),
    (["WAT"], [700], 34.0, 9.5),
])
def test_matches_oracle(species, counts, L, cutoff):
    system, r, _ = configs.build(species, counts, L, seed=6)
    if system.polar:
        d = np.random.default_rng(1).normal(scale=0.05, size=r.shape)
        d[system.qpol == 0] = 0
        r = np.vstack([r, d])
    ew = ([L] * 3, cutoff, 3.12 / cutoff, (4 + 1e-6) / L)
    fp = M.ForcePath(system, *ew, precision="fp64")
    f, e = fp.forces(r, measure=True)
    fo, eo = O.Oracle(system, *ew).forces(r, measure=True, nthreads=4)
    # FP64 both, other orders of the sums: the bounds of the FP64 path elsewhere
    assert np.sqrt(((f - fo) ** 2).sum() / (fo ** 2).sum()) < 1e-10
    assert abs(e["el"] - eo["el"]) <= 1e-10 * abs(eo["eself"])
    assert abs(e["lj"] - eo["lj"]) <= 1e-10 * abs(eo["lj"])
    assert abs(e["vir"] - eo["vir"]) <= 1e-9 * abs(eo["vir"])
    for m in range(6):
        assert abs(e["Pvir"][m] - eo["Pvir"][m]) <= 1e-9 * abs(eo["Pvir"][0])
    assert np.allclose(f, fp.forces(r)[0], rtol=0, atol=1e-12 * np.abs(fo).max())
