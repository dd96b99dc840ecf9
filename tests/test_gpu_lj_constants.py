"""The constants of the FP32 pair kernels carry no common error into the sums of
a liquid: Lennard-Jones energy and virial (terms that nearly cancel: a relative
error of sigma^2 or of the unit of length comes out some 50 times as large),
r-space energy and virial tensor against the FP64 path, over edges whose
fixed-point step rounds differently, for every pair kernel."""
import numpy as np
import pytest

import macsimus_gb300 as M
from macsimus_gb300 import configs

pytestmark = pytest.mark.gpu


def energies(species, counts, density, variant):
    L = configs.box_length(species, counts, density)
    system, r, _ = configs.build(species, counts, L, seed=5)
    rng = np.random.default_rng(6)
    r = r + rng.normal(scale=0.12, size=(system.nmol, 3))[system.mol]
    ew = ([L] * 3, 10.0, 0.31, (9 + 1e-6) / L)
    kw = dict(skin=1.0) if variant == "list" else dict(pair_variant=variant)
    e = M.ForcePath(system, *ew, kspace_engine=1, **kw).forces(r, measure=True)[1]
    return e, M.ForcePath(system, *ew, precision="fp64").forces(r, measure=True)[1]


@pytest.mark.parametrize("variant", [0, 1, 8, "list"])
@pytest.mark.parametrize("species,counts,density", [
    (["WAT"], [1500], 0.99), (["WAT"], [1500], 1.01), (["WAT"], [1500], 1.03),
    (["WAT"], [2200], 1.0), (["WAT", "NA", "CL"], [2741, 37, 37], 1.02)])
def test_sums_of_a_liquid(species, counts, density, variant):
    e, d = energies(species, counts, density, variant)
    # FP32 roundings of a pair's terms, 2^-24 some ten times over, independent from
    # pair to pair: of 1e5 pairs 50 x 10 x 6e-8 / sqrt(1e5) = 1e-7 of the virial, twice
    # that with the three constants' own; a common error of 6e-8 makes 3e-6
    assert abs(e["vir"] - d["vir"]) < 5e-7 * abs(d["vir"])
    # of the energy's two sums R - A (the virial is 12 R - 6 A), which may cancel to
    # anything: 1e-7 of R + A
    assert abs(e["lj"] - d["lj"]) < 1e-7 * (abs(d["vir"]) / 3 + 3 * abs(d["lj"]))
    # charge terms: exclusions exact to 1e-9, the others' mean error (spline_f) small
    assert abs(e["er"] - d["er"]) < 2e-8 * abs(d["er"])
    big = np.abs(d["Pvir"]).max()
    assert np.abs(np.array(e["Pvir"]) - d["Pvir"]).max() < 1e-6 * big
