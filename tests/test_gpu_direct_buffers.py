"""A context whose force evaluations run the non-uniform transforms holds the
buffers of the direct Ewald passes only once mg_ewald has run them."""
import numpy as np
import pytest

import macsimus_gb300 as M
from macsimus_gb300 import configs

pytestmark = pytest.mark.gpu


def test_direct_buffers_come_with_the_first_ewald():
    import torch
    n = 8000
    L = configs.box_length(["WAT"], [n], 0.997)
    system, r, _ = configs.build(["WAT"], [n], L, seed=2)
    ew = ([L] * 3, 12.0, 0.26, (12 + 1e-6) / L)

    def held(**kw):
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        fp = M.ForcePath(system, *ew, **kw)
        f = fp.forces(r)[0]
        torch.cuda.synchronize()
        return fp, f, free - torch.cuda.mem_get_info()[0]

    M.ForcePath(system, *ew).forces(r)          # modules loaded
    fp, f, own = held()
    direct, _, other = held(kspace_engine=3)
    # the passes' operand planes and phase rows take 40 MB here, the grids 1 MB
    assert own < other - (16 << 20)
    k, e = fp.ewald(r)
    kd, ed = direct.ewald(r)
    assert np.array_equal(k, kd) and e == ed
    assert np.array_equal(fp.ewald(r)[0], kd)
    assert np.array_equal(fp.forces(r)[0], f)
