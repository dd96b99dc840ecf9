"""Which pair kernel a box runs, and the all-pairs kernel where cells are kept
(the cutoff leaves fewer than four sites a cell): alone against the FP64 path, in
batches of its own and beside boxes on the half-shell kernel, measured and
plain, each box bit for bit as alone."""
import numpy as np
import pytest

import macsimus_gb300 as M
from macsimus_gb300 import configs

pytestmark = pytest.mark.gpu

# FP32 pair terms from exact separations (tests/test_gpu_pair_all.py)
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


def ewald(L, cutoff):
    return [L] * 3, cutoff, 3.12 / cutoff, (6 + 1e-6) / L


@pytest.mark.parametrize("species,counts,L,cutoff,kw,kernel", [
    (["WAT"], [216], 18.65, 9.0, {}, "all-pairs"),                      # one cell
    (["WAT"], [216], 18.65, 9.0, dict(pair_variant=8), "all-pairs"),
    (["WAT"], [300], 26.0, 11.8, {}, "all-pairs"),                      # 1331 cells
    (["WAT"], [300], 26.0, 11.8, dict(pair_variant=9), "half-shell"),
    (["WAT"], [300], 26.0, 9.0, {}, "half-shell"),                      # 125 cells
    (["WAT"], [300], 26.0, 9.0, dict(pair_variant=10), "half-shell"),
    (["WAT"], [300], 26.0, 9.0, dict(pair_variant=8), "group"),
    (["WAT"], [300], 26.0, 9.0, dict(pair_variant=3), "cell"),
    (["WAT"], [300], 26.0, 9.0, dict(precision="fp64"), "fp64"),
    (["WAT"], [300], 26.0, 9.0, dict(skin=1.0), "list"),
    (["WAT"], [864], 29.65, 12.0, {}, "half-shell"),                    # 343 cells
    (["T4P"], [1024], 31.4, 11.0, {}, "half-shell"),                    # 125 cells
])
def test_which_kernel(species, counts, L, cutoff, kw, kernel):
    system, r, _ = box(species, counts, L)
    fp = M.ForcePath(system, *ewald(L, cutoff), **kw)
    assert fp.pair_kernel == kernel
    fd = M.ForcePath(system, *ewald(L, cutoff), precision="fp64").forces(r)[0]
    assert rel(fp.forces(r)[0], fd) < (1e-12 if kernel == "fp64" else TOL)


@pytest.mark.parametrize("species,counts,L,cutoff", [
    (["NA", "CL"], [8, 8], 25.0, 11.5),        # 16 sites: half a batch of neighbours
    (["NA", "CL"], [17, 16], 25.0, 11.5),      # one site past a batch
    (["WAT"], [171], 24.0, 10.9),              # 513: one past 16 batches
    (["WATD"], [190], 24.0, 10.9),             # shells
    (["T4P"], [300], 26.0, 11.8),              # sites without charge or LJ
    (["WAT"], [700], 30.0, 13.9),
])
def test_all_pairs_over_kept_cells_match_fp64(species, counts, L, cutoff):
    system, r, _ = box(species, counts, L)
    fp = M.ForcePath(system, *ewald(L, cutoff))
    assert fp.pair_kernel == "all-pairs"
    f, e = fp.forces(r, measure=True)
    fd, ed = M.ForcePath(system, *ewald(L, cutoff), precision="fp64").forces(r, measure=True)
    assert rel(f, fd) < TOL
    assert abs(e["er"] - ed["er"]) < 1e-6 * abs(ed["eself"])
    assert np.array_equal(f, fp.forces(r)[0])


ALL = [(["WAT"], [300], 26.0, 11.8), (["WAT"], [171], 24.0, 10.9), (["NA", "CL"], [17, 16], 25.0, 11.5)]
HALF = [(["WAT"], [300], 26.0, 9.0), (["WAT"], [700], 34.0, 9.0)]


@pytest.mark.parametrize("measure", [True, False])
@pytest.mark.parametrize("boxes", [ALL, [ALL[0], HALF[1]], [HALF[0], ALL[2], HALF[1], ALL[1]]],
                         ids=["all-pairs", "one of each", "mixed"])
def test_batches(boxes, measure):
    arg = []
    for s, n, L, rc in boxes:
        system, r, r1 = box(s, n, L)
        ew = ewald(L, rc)
        arg.append((dict(system=system, L=ew[0], cutoff=rc, alpha=ew[2], kappa=ew[3], h=0.001), r, r1))
    batch = M.Batch([a[0] for a in arg], lanes=2)
    for fp, b in zip(batch.box, boxes):
        assert fp.pair_kernel == ("all-pairs" if b in ALL else "half-shell")
    for fp, (_, r, r1) in zip(batch.box, arg):
        fp.md_set_state(r, r1)
    en = batch.md_steps(3, measure=measure)
    assert batch.fused
    for i, (a, r, r1) in enumerate(arg):
        a = dict(a)
        fp = M.ForcePath(a.pop("system"), a.pop("L"), a.pop("cutoff"), a.pop("alpha"),
                         a.pop("kappa"), **a)
        fp.md_set_state(r, r1)
        e1 = fp.md_steps(3, measure=measure)
        assert np.array_equal(batch.box[i].md_get_state()[0], fp.md_get_state()[0])
        assert np.array_equal(batch.box[i].md_get_state()[1], fp.md_get_state()[1])
        if measure:
            assert en[i]["el"] == e1["el"] and en[i]["Ptens"] == e1["Ptens"]
    batch.close()
