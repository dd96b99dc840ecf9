"""The Ewald k-space sums of the FP32 path as non-uniform transforms (the
automatic engine) against the FP64 sums and the direct FP32 sums: grids from
the smallest (16 points an edge, the window as wide as half of it) to one of
more than 100 points, edges of different length, partial tiles, uncharged
sites, shells beyond the margin of the cell lookup, one cell for the box."""
import numpy as np
import pytest

import macsimus_gb300 as M
from macsimus_gb300 import configs, forcefield as ff

pytestmark = pytest.mark.gpu

# relative to the k-space force RMS.  Transforms: window 5e-7 and FP32
# arithmetic 8e-7; direct FP32 sums: 2.4e-6 on 98304 sites.  Twice their sum
# of squares' root covers the few-charge boxes, whose sums average less.
TOL = 5e-6

CASES = {
    # name: species, counts, edges, cutoff, alpha, largest |n| along x
    "one_cell": (["WAT"], [190], (18.1, 18.1, 18.1), 9.0, 0.40, 5),
    "tiny_k": (["WAT"], [216], (18.7, 18.7, 18.7), 9.0, 0.12, 2),
    "uneven": (["WAT"], [600], (19.0, 24.5, 39.3), 9.0, 0.35, 7),
    "ions": (["WAT", "NA", "CL"], [500, 9, 9], (25.3, 25.3, 25.3), 10.0, 0.31, 9),
    "uncharged": (["T4P"], [300], (21.0, 21.0, 21.0), 9.0, 0.35, 6),
    "fine": (["WAT"], [432], (23.6, 23.6, 23.6), 9.0, 1.0, 30),
}


def box(case, seed=3):
    species, counts, edges, cutoff, alpha, kn = CASES[case]
    system, r, r1 = configs.build(species, counts, min(edges), seed=seed)
    # the lattice of the shortest edge, stretched to the box molecule by molecule
    shift = np.zeros((system.nmol, 3))
    first = r[system.mol_first[:-1]]
    for d in range(3):
        shift[:, d] = first[:, d] * (edges[d] / min(edges) - 1)
    r = r + shift[system.mol]
    return system, r, edges, cutoff, alpha, (kn + 1e-6) / edges[0]


def rms(a):
    return float(np.sqrt((a ** 2).sum()))


@pytest.mark.parametrize("case", sorted(CASES))
def test_transforms_match_the_direct_sums(case):
    system, r, *ew = box(case)
    f0, e0 = M.ForcePath(system, *ew).forces(r, measure=True)
    f1, e1 = M.ForcePath(system, *ew, kspace_engine=1).forces(r, measure=True)
    p64 = M.ForcePath(system, *ew, precision="fp64")
    f64, e64 = p64.forces(r, measure=True)
    fk, _ = p64.ewald(r)
    assert rms(f0 - f1) < TOL * rms(fk)
    assert abs(e0["ek"] - e64["ek"]) < 2e-6 * e64["ek"]
    # the k-space part of the virial tensor (the rest is the same arithmetic)
    d = np.array(e0["Pvir"]) - np.array(e1["Pvir"])
    assert np.abs(d).max() < 5e-6 * e64["ek"]
    # the measured and the plain evaluation move the sites identically
    assert np.array_equal(f0, M.ForcePath(system, *ew).forces(r)[0])


@pytest.mark.parametrize("reach", [0.05, 0.49, 0.9])
def test_shells_near_and_far_from_their_sites(reach):
    """Drude displacements within the lookup margin (0.5 A), at its edge and
    beyond it (every tile then scans the box)"""
    n = 400
    L = configs.box_length(["WATD"], [n], 0.997)
    system, r, _ = configs.build(["WATD"], [n], L, seed=4)
    rng = np.random.default_rng(5)
    d = rng.uniform(-1, 1, r.shape) * reach
    d[system.qpol == 0] = 0
    r = np.vstack([r, d])
    ew = ([L] * 3, 10.0, 0.31, (7 + 1e-6) / L)
    f0, e0 = M.ForcePath(system, *ew).forces(r, measure=True)
    f1, e1 = M.ForcePath(system, *ew, kspace_engine=1).forces(r, measure=True)
    p64 = M.ForcePath(system, *ew, precision="fp64")
    fk, _ = p64.ewald(r)
    e64 = p64.forces(r, measure=True)[1]
    assert rms(f0 - f1) < TOL * rms(fk)
    assert abs(e0["ek"] - e64["ek"]) < 2e-6 * e64["ek"]
