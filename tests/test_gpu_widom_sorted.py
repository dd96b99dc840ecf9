"""Insertions sorted by place (many per cell) against a warp per insertion
(few per cell): the energy of insertion k depends on the seed and k alone, so
a call of few insertions gives the values that a call of many must repeat;
one and several sites, charged and not, coarse and fine cells, past the
workspace's limit."""
import numpy as np
import pytest

import macsimus_gb300 as M
from macsimus_gb300 import configs
from macsimus_gb300 import forcefield as ff

pytestmark = pytest.mark.gpu

PRB = ff.TYPE_ORDER.index("PRB")
T = 298.0
GAMMA = 0x9E3779B97F4A7C15   # the stream's step per word, 8 words an insertion


def close(a, b):
    """FP32 terms either way, added in other groups: 1e-6 of the energy, and of
    the cancelling terms of a charged ghost (about 1e5 K)"""
    return (np.abs(a - b) <= 1e-6 * np.abs(b) + 0.2).all()


@pytest.mark.parametrize("counts,L,cells", [(60, 22.0, 1), (60, 22.0, 2), (300, 34.0, 2)])
@pytest.mark.parametrize("nps,charged", [(1, False), (1, True), (3, True), (8, False)])
def test_same_energies_on_both_paths(counts, L, cells, nps, charged):
    system, r, _ = configs.build(["NA", "CL"], [counts, counts], L, seed=2)
    fp = M.ForcePath(system, [L] * 3, 10.9, 0.29, (5 + 1e-6) / L, cells_per_cutoff=cells)
    fp.forces(r)
    rng = np.random.default_rng(nps)
    g = rng.uniform(-1, 1, (nps, 3)) if nps > 1 else np.zeros((1, 3))
    q = rng.uniform(-0.5, 0.5, nps) if charged else None
    kw = dict(geometry=g, charges=q, seed=77, T=T, energies=True)
    few = fp.widom([PRB] * nps, n=3, **kw)
    for n in (24601, 70000):
        many = fp.widom([PRB] * nps, n=n, **kw)
        assert close(many["U"][:3], few["U"])
        # another number of neighbours, the same values
        assert np.array_equal(many["U"][:24601], fp.widom([PRB] * nps, n=24601, **kw)["U"])
        e = -many["U"] / T
        assert many["sum"] == pytest.approx(np.exp(e[e > -700]).sum(), rel=1e-12)


def test_several_chunks():
    system, r, _ = configs.build(["NA", "CL"], [60, 60], 22.0, seed=2)
    fp = M.ForcePath(system, [22.0] * 3, 10.9, 0.29, (5 + 1e-6) / 22.0)
    fp.forces(r)
    # 40008 sites behind the limit
    nps, cn = 8, (1 << 23) // 8
    g = np.random.default_rng(1).uniform(-0.5, 0.5, (nps, 3))
    n = cn + 5001
    res = fp.widom([PRB] * nps, geometry=g, n=n, seed=9, T=T, energies=True)
    tail = fp.widom([PRB] * nps, geometry=g, n=5001, seed=(9 + 8 * cn * GAMMA) % 2 ** 64, T=T,
                    energies=True)
    assert np.array_equal(res["U"][cn:], tail["U"])
    e = -res["U"] / T
    assert res["sum"] == pytest.approx(np.exp(e[e > -700]).sum(), rel=1e-12)
