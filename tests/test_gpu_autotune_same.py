"""The autotuner does not choose between choices that come to the same
evaluation: they share one timing, and a split that nothing reads stays the
caller's."""
import numpy as np
import pytest

import macsimus_gb300 as M
from golden_cases import load

pytestmark = pytest.mark.gpu


def tune(**kw):
    g, _, system, ew = load("spce864")
    return M.autotune(system, ew["L"], ew["cutoff"], ew["alpha"], ew["kappa"], g["r"][0], **kw)


def test_transforms_read_no_split():
    best = tune(kspace_ctas_per_sm=7)
    assert (best["ms"] == best["ms"][:, :1]).all()
    assert best["kspace_ctas_per_sm"] == 7
    assert tune()["kspace_ctas_per_sm"] == 10


def test_direct_sums_time_the_split():
    best = tune(kspace_engine=1)
    assert (best["ms"] != best["ms"][:, :1]).any()
    assert best["kspace_ctas_per_sm"] in (6, 10, 16)


def test_one_kernel_one_timing():
    best = tune()
    assert np.array_equal(best["ms_half"], best["ms_half_t"])
    # pair_variant 0 is the half-shell kernel here
    assert best["ms_pair"][0] in best["ms_half"]
    # a box held in one cell runs all pairs whatever the variant
    g, _, system, ew = load("spce216")
    one = M.autotune(system, ew["L"], ew["cutoff"], ew["alpha"], ew["kappa"], g["r"][0])
    assert M.ForcePath(system, ew["L"], ew["cutoff"], ew["alpha"], ew["kappa"]).pair_kernel == "all-pairs"
    assert (one["ms_pair"] == one["ms_pair"][0]).all() and one["pair_variant"] == 0


def test_fp64_has_one_pair_kernel():
    best = tune(precision="fp64")
    assert (best["ms_pair"] == best["ms_pair"][0]).all()
    assert (best["ms"] == best["ms"][:, :1]).all()
