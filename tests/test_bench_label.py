"""bench.py names the pair kernel that ran: every kernel the library may report
has its label, and no label stands for two."""
import os
import re

import bench

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_pair_kernel_has_its_own_label():
    src = open(os.path.join(REPO, "macsimus_gb300", "csrc", "mg_api.cu")).read()
    body = src[src.index("const char* mg_pair_kernel("):]
    names = set(re.findall(r'"([a-z0-9-]+)"', body[:body.index("\n}")]))
    assert names == set(bench.PAIR_LABEL)
    assert len(set(bench.PAIR_LABEL.values())) == len(names)
