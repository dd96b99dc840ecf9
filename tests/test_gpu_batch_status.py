"""A measured step of a batch reports what an unmeasured one does: a position
that is not finite, SHAKE that does not converge."""
import numpy as np
import pytest

import macsimus_gb300 as M
from macsimus_gb300 import configs

pytestmark = pytest.mark.gpu


def batch(n=300, L=26.0, **kw):
    system, r, r1 = configs.build(["WAT"], [n], L, seed=5)
    kw = dict(L=[L] * 3, cutoff=9.0, alpha=0.35, kappa=(7 + 1e-6) / L, **kw)
    b = M.Batch([dict(system=system, **kw) for _ in range(2)])
    for fp in b.box:
        fp.md_set_state(r, r1)
    return b, r, r1


@pytest.mark.parametrize("measure", [True, False])
def test_non_finite_position(measure):
    b, r, r1 = batch()
    r = r.copy()
    r[7, 1] = np.nan
    b.box[1].md_set_state(r, r1)
    with pytest.raises(M.MGError, match="box 1: non-finite"):
        b.md_steps(1, measure=measure)
    b.close()


@pytest.mark.parametrize("measure", [True, False])
def test_shake_not_converged(measure):
    b, r, r1 = batch(shake_maxit=1, epsc=1e-12)
    with pytest.raises(M.MGError, match="SHAKE"):
        b.md_steps(1, measure=measure)
    b.close()
