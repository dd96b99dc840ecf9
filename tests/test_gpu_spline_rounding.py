"""The coefficients of the FP32 erfc splines leave no common error on the pairs: the
charge part of the trace of 864 waters' virial tensor, whose terms of either sign add
up to 2e-5 of their size, over eight configurations against the FP64 path."""
import numpy as np
import pytest

import macsimus_gb300 as M
from macsimus_gb300 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 1])
def test_no_common_error_of_the_charge_terms(variant):
    L = 29.65
    ew = ([L] * 3, 12.0, 0.26, (8 + 1e-6) / L)
    off = []
    for seed in range(8):
        system, r, _ = configs.build(["WAT"], [864], L, seed=seed)
        system.typeE[:] = 0
        rng = np.random.default_rng(seed)
        r = r + rng.normal(scale=0.12, size=(system.nmol, 3))[system.mol]
        e = M.ForcePath(system, *ew, kspace_engine=1, pair_variant=variant).forces(r, measure=True)[1]
        d = M.ForcePath(system, *ew, precision="fp64").forces(r, measure=True)[1]
        off.append(sum(e["Pvir"][:3]) - sum(d["Pvir"][:3]))
    # some 9e5 pairs within the cutoff, 900 K each on the average and a few 1e4 K the
    # closest, to 2^-24: about 0.4 K a configuration; a common error of one 2^-24 of
    # the closest alone makes 5 K
    assert abs(np.mean(off)) < 3 * 0.4 / np.sqrt(8)
