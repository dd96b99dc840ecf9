"""The FP32 pair kernels read the erfc spline's interval that holds r^2, in its upper
half too: two charges at places of their intervals against the FP64 path."""
import numpy as np
import pytest

import macsimus_gb300 as M
from macsimus_gb300 import configs

pytestmark = pytest.mark.gpu

ALPHA, GRID = 0.31, 256      # intervals of alpha^2 r^2


@pytest.mark.parametrize("kw", [{}, dict(pair_variant=1), dict(pair_variant=8), dict(skin=1.0)],
                         ids=["half-shell", "cell", "group", "list"])
@pytest.mark.parametrize("interval", [10, 16, 24, 36])        # 0.65 to 1.2 A
@pytest.mark.parametrize("place", [0.25, 0.52, 0.75])
def test_two_charges(interval, place, kw):
    system, _, _ = configs.build(["NA", "CL"], [1, 1], 40.0, seed=1)
    system.typeE[:] = 0
    r = np.array([[20.0, 20.0, 20.0]] * 2)
    r[1, 0] += np.sqrt((interval + place) / GRID) / ALPHA
    ew = ([40.0] * 3, 10.0, ALPHA, (3 + 1e-6) / 40.0)

    def forces(**k):
        fp = M.ForcePath(system, *ew, **k)
        return (fp.forces(r)[0] - fp.ewald(r)[0])[0, 0]
    f, f64 = forces(kspace_engine=1, **kw), forces(precision="fp64")
    # roundings of r^2, of the three coefficients, of the denominator, its reciprocal
    # (two 2^-24) and the sum, three times over where the terms are larger than it
    assert abs(f - f64) < 24 * 2.0 ** -24 * abs(f64)
