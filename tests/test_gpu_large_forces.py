"""Forces beyond the range of the half-shell kernel's fixed-point sums (2^31
K/A): overlapping sites of a random start get their forces, coincident ones
give a non-finite force and the error it leads to, in single evaluations, MD
steps and batches; the evaluation after is as if nothing had happened."""
import numpy as np
import pytest

import macsimus_gb300 as M
from macsimus_gb300 import configs

pytestmark = pytest.mark.gpu

L, CUTOFF = 29.65, 12.0
EWALD = ([L] * 3, CUTOFF, 0.26, (8 + 1e-6) / L)
# the 13th power of a separation good to a few 2^-24, the reciprocal's rounding
TOL_PAIR = 1e-5
# all forces of an ordinary evaluation: FP32 pair terms (tests/test_gpu_pair_all.py)
TOL = 3e-6


def box(gap, species="WAT", seed=3):
    """864 waters, the second one moved so that the oxygens are gap apart"""
    system, r, r1 = configs.build([species], [864], L, seed=seed)
    a, b, c = (int(system.mol_first[m]) for m in (0, 1, 2))
    if gap is not None:
        r[b:c] += r[a] + [gap, 0.01 * gap, 0.0] - r[b]
    if system.polar:
        d = np.random.default_rng(seed).normal(scale=0.02, size=r.shape)
        d[system.qpol == 0] = 0
        r, r1 = np.vstack([r, d]), np.vstack([r1, 0 * r1])
    return system, r, r1, [a, b]


def rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


@pytest.mark.parametrize("species", ["WAT", "WATD"])
@pytest.mark.parametrize("gap", [1.05, 0.9, 0.6, 0.3])   # 2e9, 1.5e10, 3e12, 2e16 K/A
def test_overlapping_pair_matches_fp64(species, gap):
    system, r, _, pair = box(gap, species)
    fp = M.ForcePath(system, *EWALD)
    f, en = fp.forces(r, measure=True)
    fd, ed = M.ForcePath(system, *EWALD, precision="fp64").forces(r, measure=True)
    assert rel(f[pair], fd[pair]) < TOL_PAIR
    rest = np.setdiff1d(np.arange(len(f)), pair)
    # the others, some of them charges a fraction of an A apart, where the FP32
    # spline is good to 1e-3 only: as the group kernel, which keeps no such sums,
    # each site's few dozen FP32 roundings aside
    f8 = M.ForcePath(system, *EWALD, pair_variant=8).forces(r)[0]
    size = np.abs(fd[rest]).max()
    assert np.abs(f[rest] - f8[rest]).max() < 32 * 2.0 ** -24 * size
    assert np.abs(f[rest] - fd[rest]).max() < 1.1 * np.abs(f8[rest] - fd[rest]).max() + 32 * 2.0 ** -24 * size
    assert abs(en["lj"] - ed["lj"]) < TOL_PAIR * abs(ed["lj"])
    # measured and plain evaluations, and a repeat, are the same bit for bit
    assert np.array_equal(f, fp.forces(r)[0])
    # and the next configuration is not touched by it
    r2 = box(None, species)[1]
    assert np.array_equal(fp.forces(r2)[0], M.ForcePath(system, *EWALD).forces(r2)[0])


def test_crowded_cell():
    """2744 weak charges 0.7 A apart in one cell: no term is large, but more
    groups than the sums have room for the terms of"""
    system, r, _ = configs.build(["NA", "CL"], [1372, 1372], 60.0, seed=2)
    system.typeE[:] = 0
    system.q *= 0.1
    i = np.arange(14)
    rng = np.random.default_rng(4)
    r = (30.5 + 0.7 * np.stack(np.meshgrid(i, i, i), -1).reshape(-1, 3))[rng.permutation(2744)]
    r = r + rng.normal(scale=0.05, size=r.shape)
    ew = ([60.0] * 3, 10.0, 0.31, (8 + 1e-6) / 60.0)
    f = M.ForcePath(system, *ew, cells_per_cutoff=1).forces(r)[0]
    fd = M.ForcePath(system, *ew, precision="fp64").forces(r)[0]
    # a force is some 10 times smaller than the sum of its pairs' magnitudes
    assert rel(f, fd) < 10 * TOL


@pytest.mark.parametrize("species", ["WAT", "WATD"])
def test_coincident_sites_give_the_error(species):
    system, r, r1, pair = box(0.0, species)
    fp = M.ForcePath(system, *EWALD)
    assert not np.isfinite(fp.forces(r)[0][pair]).any()
    fp.md_set_state(r, r1)
    with pytest.raises(M.MGError, match="non-finite"):
        fp.md_steps(3)


def run_one(system, r, r1, steps, **kw):
    fp = M.ForcePath(system, *EWALD, h=1e-7, **kw)
    fp.md_set_state(r, r1)
    fp.md_steps(steps)
    return fp.md_get_state()[0]


def test_md_step_moves_an_overlapping_pair_apart():
    system, r, r1, pair = box(0.9)
    r1 = 0 * r1
    d0 = run_one(system, r, r1, 2) - r
    d8 = run_one(system, r, r1, 2, pair_variant=8) - r
    assert np.abs(d8[pair]).max() > 1e-8
    # differences of positions of some 30 A in FP64
    assert np.abs(d0[pair] - d8[pair]).max() < 1e-4 * np.abs(d8[pair]).max()


def test_batch():
    """an overlapping and an ordinary box in a batch: each as alone; a box with
    coincident sites: the error"""
    arg = dict(L=EWALD[0], cutoff=CUTOFF, alpha=EWALD[2], kappa=EWALD[3], h=1e-7)
    bs = [box(g) for g in (0.9, None)]
    batch = M.Batch([dict(system=b[0], **arg) for b in bs], lanes=2)
    for fp, b in zip(batch.box, bs):
        fp.md_set_state(b[1], 0 * b[2])
    batch.md_steps(2)
    assert batch.fused
    for fp, b in zip(batch.box, bs):
        assert np.array_equal(fp.md_get_state()[0], run_one(b[0], b[1], 0 * b[2], 2))
    c = box(0.0)
    batch.box[1].md_set_state(c[1], 0 * c[2])
    with pytest.raises(M.MGError, match="non-finite"):
        batch.md_steps(3, measure=False)
    batch.close()
