"""Both sides of the rules that pick a kernel: no index outside a field in the bounds-checked build
(tests/checked_dispatch.py), and the heatbath of both against the oracle at ragged sizes."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_no_out_of_bounds_access():
    r = subprocess.run([sys.executable, os.path.join(HERE, "checked_dispatch.py")], capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-4000:]
    report = json.loads(r.stdout.strip().splitlines()[-1])
    assert report["checked"] is True
    assert report["count"] == 0, hex(report["first"])


@pytest.mark.parametrize("L", [(14, 10, 6, 4), (14, 10, 6, 6)])  # 1680 and 2520 links a set: the small kernel, the other
def test_heatbath_sets_match_the_oracle(gpu, orc, L):
    """Each (parity, mu) set from the same input, FP64, to the 1e-12 of the parity tests."""
    U = orc.hot_start(L, 7)
    f = gpu.GaugeField(L, 64, 0)
    for par in range(2):
        for mu in range(4):
            f.upload(U)
            V = U.copy()
            f.hb_subsweep(5.9, 2, 31, 4, par, mu)
            orc.hb_subsweep(V, L, 5.9, 2, 31, 4, par, mu)
            assert np.max(np.abs(f.download() - V)) < 1e-12, (par, mu)
