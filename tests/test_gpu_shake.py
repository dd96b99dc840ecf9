"""SHAKE's paths for three constrained sites (constraints in the order (0,1),
(0,2), (1,2); in another order; with a massless fourth site behind them) and
the general one, at molecule counts around its 32 molecules per CTA: one step
against the oracle's, and the paths against each other."""
import copy

import numpy as np
import pytest

import macsimus_gb300 as M
from macsimus_gb300 import configs
from oracle import oracle as O

pytestmark = pytest.mark.gpu

EPS = 1e-10
# a sweep more or fewer where |d| meets its limit to rounding: three
# constraints of up to 1.6 A, each moved by less than eps times its length
TOL = 3 * 1.6 * EPS


def permuted(system):
    s = copy.deepcopy(system)
    for n in range(s.nmol):
        c0, c1 = s.mol_cfirst[n], s.mol_cfirst[n + 1]
        if c1 - c0 == 3:
            s.cons[c0:c1] = s.cons[[c0 + 2, c0, c0 + 1]][:, ::-1]
            s.cons_len[c0:c1] = s.cons_len[[c0 + 2, c0, c0 + 1]]
    return s


def step(system, L, r, r1, precision, measure=True):
    fp = M.ForcePath(system, [L] * 3, 9.0, 0.34, (5 + 1e-6) / L, precision=precision, h=0.001,
                     epsc=EPS)
    f, _ = fp.forces(r)
    fp.md_set_state(r, r1)
    en = fp.md_steps(1, measure=measure)
    return f, fp.md_get_state(), en


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("species,counts,order", [
    (["WAT"], [31], "plain"), (["WAT"], [32], "plain"), (["WAT"], [33], "permuted"),
    (["NA", "WAT", "CL"], [2, 65, 2], "plain"), (["NA", "WAT", "CL"], [2, 65, 2], "permuted"),
])
def test_step_matches_oracle(species, counts, order, precision):
    L = 20.0
    system, r, r1 = configs.build(species, counts, L, seed=3, h=0.001)
    if order == "permuted":
        system = permuted(system)
    f, (rg, vg), en = step(system, L, r, r1, precision)
    meas = np.zeros(13)
    ro, vo, _, ekin = O.Oracle(system, [L] * 3, 9.0, 0.34, (5 + 1e-6) / L).shake_step(
        r, r1, f, 0.001, eps=EPS, omega=0.6, meas=meas)
    d = rg - ro
    d -= L * np.round(d / L)          # positions are wrapped after the step
    assert np.abs(d).max() < TOL
    assert np.abs(vg - vo).max() < TOL
    assert en["ekin"] == pytest.approx(ekin, rel=1e-7)
    assert np.array_equal(rg, step(system, L, r, r1, precision, measure=False)[1][0])


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_massless_fourth_site(precision):
    # in another order of its constraints a four-site water takes the general path
    L = 20.0
    system, r, r1 = configs.build(["T4P", "NA", "CL"], [64, 1, 1], L, seed=4, h=0.001)
    _, (ra, va), ea = step(system, L, r, r1, precision)
    _, (rb, vb), eb = step(permuted(system), L, r, r1, precision)
    # the sweeps approach the solution from other sides: to within the limit
    # over the slowest contraction of a sweep (omega 0.6: less than 1/2)
    assert np.abs(ra - rb).max() < 4 * TOL
    assert np.abs(va - vb).max() < 4 * TOL
    assert ea["ekin"] == pytest.approx(eb["ekin"], rel=1e-6)
