"""The all-pairs kernel of small boxes (one cell, or filled by the cutoff
sphere): site counts around its batches of 32 sites and its 16 warps, Drude
shells, against the FP64 path; the measured and the plain evaluation give the
same forces; a batch gives each box what it gets alone."""
import numpy as np
import pytest

import macsimus_gb300 as M
from macsimus_gb300 import configs

pytestmark = pytest.mark.gpu

# FP32 pair terms from exact separations, as the cell kernels: each within a
# few 1e-7 of its FP64 value, LJ cores (12th powers) within 1e-6
TOL = 3e-6


def rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


def box(species, counts, L, seed=8):
    system, r, r1 = configs.build(species, counts, L, seed=seed)
    if system.polar:
        d = np.random.default_rng(seed).normal(scale=0.05, size=r.shape)
        d[system.qpol == 0] = 0
        r = np.vstack([r, d])
    return system, r, r1


@pytest.mark.parametrize("species,counts,L,cutoff", [
    (["NA", "CL"], [8, 8], 22.0, 10.9),          # 16 sites: half a batch, one cell
    (["NA", "CL"], [16, 16], 22.0, 10.9),        # exactly one batch
    (["WAT"], [11], 22.0, 10.9),                 # 33: one site into the second
    (["WAT"], [171], 18.2, 9.0),                 # 513: one site past 16 batches
    (["WATD"], [190], 18.2, 9.0),                # shells, one cell
    (["WAT"], [864], 29.65, 12.0),               # cells kept for the k-space sums
    (["T4P"], [1024], 31.4, 11.0),               # 4096 sites, uncharged ones among them
])
def test_all_pairs_match_fp64(species, counts, L, cutoff):
    system, r, _ = box(species, counts, L)
    ew = ([L] * 3, cutoff, 3.12 / cutoff, (6 + 1e-6) / L)
    f0, e0 = M.ForcePath(system, *ew).forces(r, measure=True)
    fd, ed = M.ForcePath(system, *ew, precision="fp64").forces(r, measure=True)
    assert rel(f0, fd) < TOL
    assert abs(e0["er"] - ed["er"]) < 1e-6 * abs(ed["eself"])
    # a sum of large terms of both signs
    assert abs(e0["lj"] - ed["lj"]) <= 1e-5 * abs(ed["lj"]) + 1e-7 * abs(ed["eself"])
    assert np.array_equal(f0, M.ForcePath(system, *ew).forces(r)[0])


def test_batched_with_cell_boxes():
    """a batch of a box on the all-pairs kernel and one on the cell kernel"""
    bs = []
    for n, L, rc in ((300, 26.0, 9.0), (700, 34.0, 9.0)):
        system, r, r1 = box(["WAT"], [n], L)
        bs.append((dict(system=system, L=[L] * 3, cutoff=rc, alpha=3.12 / rc,
                        kappa=(7 + 1e-6) / L, h=0.001), r, r1))
    batch = M.Batch([b[0] for b in bs], lanes=2)
    for fp, (_, r, r1) in zip(batch.box, bs):
        fp.md_set_state(r, r1)
    en = batch.md_steps(3)
    assert batch.fused
    for i, (a, r, r1) in enumerate(bs):
        a = dict(a)
        fp = M.ForcePath(a.pop("system"), a.pop("L"), a.pop("cutoff"), a.pop("alpha"),
                         a.pop("kappa"), **a)
        fp.md_set_state(r, r1)
        e1 = fp.md_steps(3)
        assert np.array_equal(batch.box[i].md_get_state()[0], fp.md_get_state()[0])
        assert en[i]["el"] == e1["el"] and en[i]["Ptens"] == e1["Ptens"]
    batch.close()
