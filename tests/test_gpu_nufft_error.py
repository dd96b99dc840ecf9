"""The k-space forces of the automatic engine (non-uniform transforms) are as
close to the 64-bit sums as those of the direct tensor-core passes, which it
stands in for: crystals with displaced molecules, the grids' smallest and largest
points per mode, k sets cut short and not, ions, shells."""
import numpy as np
import pytest

import macsimus_gb300 as M
from macsimus_gb300 import configs

pytestmark = pytest.mark.gpu

BOXES = {
    # species, counts, density, cutoff, alpha, largest |n|
    "water_216": (["WAT"], [216], 0.997, 9.0, 0.35, 7),
    "brine_12": (["WAT", "NA", "CL"], [4096, 128, 128], 1.06, 10.0, 0.31, 12),
    "brine_20": (["WAT", "NA", "CL"], [12503, 254, 254], 1.0464, 10.076, 0.3096, 20),
    "cut_short": (["WAT", "NA", "CL"], [24000, 800, 800], 1.05, 9.5, 0.3284, 20),
    "water_20": (["WAT"], [23812], 0.9955, 10.481, 0.2977, 20),
    "shells": (["WATD"], [3000], 0.997, 12.0, 0.26, 9),
}


def rms(a):
    return float(np.sqrt((a ** 2).mean()))


@pytest.mark.parametrize("name", sorted(BOXES))
def test_no_further_from_the_64_bit_sums_than_the_direct_passes(name):
    species, counts, density, cutoff, alpha, kn = BOXES[name]
    L = configs.box_length(species, counts, density)
    system, r, _ = configs.build(species, counts, L, seed=11)
    rng = np.random.default_rng(12)
    r = r + rng.normal(scale=0.12, size=(system.nmol, 3))[system.mol]
    if system.polar:
        d = rng.normal(scale=0.05, size=r.shape)
        d[system.qpol == 0] = 0
        r = np.vstack([r, d])
    ew = ([L] * 3, cutoff, alpha, (kn + 1e-6) / L)
    k64 = M.ForcePath(system, *ew, precision="fp64").ewald(r)[0]
    direct = M.ForcePath(system, *ew, kspace_engine=3)
    f3, k3 = direct.forces(r)[0], direct.ewald(r)[0]
    # the r-space parts are the same bit for bit
    k0 = M.ForcePath(system, *ew).forces(r)[0] - f3 + k3
    assert rms(k0 - k64) <= rms(k3 - k64)
