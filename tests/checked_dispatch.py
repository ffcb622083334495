"""libqcb_checked.so on both sides of the rules that pick a kernel, as one JSON line (the out-of-bounds record).

Run in a process of its own, as checked_workload.py; tests/test_gpu_checked_dispatch.py asserts on the output.
The lattices lie on either side of the line of the small lattices' heatbath (2368 links a set), none a multiple of
a block's links or of a tile; every storage is copied into every other.
"""
import json
import os
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)

from conftest import load_package  # noqa: E402

FORMATS = [(64, 0), (64, 1), (32, 0), (32, 1)]
SHAPES = [(2, 2, 6, 2), (14, 10, 6, 4), (14, 10, 6, 6)]  # 24, 1680 and 2520 half-sites


def main():
    qcb = load_package()
    qcb.load_library(qcb.CHECKED_LIB_PATH)
    checked, _, _ = qcb.debug_oob()
    for L in SHAPES:
        fields = [qcb.GaugeField(L, *fmt) for fmt in FORMATS]
        for f in fields:
            f.hot_start(3)
            for n_hits in (0, 1, 3):
                f.hb_sweep(5.7, n_hits, 1, n_hits)
            f.hb_sweep(0.5, 2, 1, 9)
            f.plaquette()
            f.clover_qe()
            fl = qcb.GradientFlow(f, 0.02)
            fl.measure(f, 3, 2, plaquette=True)
            fl.measure(f, 2, 0)
            fl.close()
        for src in fields:
            for dst in fields:
                dst.copy_from(src)
        for f in fields:
            f.unitarity()
            f.close()
    _, count, first = qcb.debug_oob()
    print(json.dumps({"checked": checked, "count": count, "first": first}))


if __name__ == "__main__":
    main()
