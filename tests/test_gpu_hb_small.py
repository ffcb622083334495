"""The small lattices' heatbath kernel (eight lanes a link) against the one-thread kernels.

A one-chain batch runs the tile kernel, one thread a link, on the same streams; the small kernel forms
every value by the same operations, so the links are equal.  Lattices below, at and past the blocks'
16 links and both sides of the line between the kernels (7104 links a set); hits from none to more
than the kernel's table of draws holds.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LATTICES = [(2, 2, 2, 2), (2, 2, 6, 2), (6, 10, 2, 2), (4, 4, 4, 4), (6, 6, 6, 6), (12, 12, 12, 8), (14, 12, 12, 8)]


@pytest.mark.parametrize("L", LATTICES)
@pytest.mark.parametrize("store", [0, 1])
@pytest.mark.parametrize("n_hits", [0, 1, 2, 5])
def test_small_lattice_sweeps_equal_the_batch(gpu, L, store, n_hits):
    f = gpu.GaugeField(L, 64, store)
    f.hot_start(11)
    b = gpu.Batch([L], [5.9], [77], 64, store)
    b.upload(0, f.download())
    f.upload(f.download())
    for sweep in range(3):
        f.hb_sweep(5.9, n_hits, 77, sweep)
    b.sweep(n_hits, 3)
    b.sync()
    assert np.array_equal(f.download(), b.download(0))


def test_small_lattice_rejections_match_the_oracle(gpu, orc):
    """A weak coupling makes most Kennedy-Pendleton attempts fail, so that links run past their table of
    draws again and again: one (parity, mu) set from the same input, to the parity tests' 1e-12."""
    L = (4, 6, 2, 8)
    U = orc.hot_start(L, 3)
    f = gpu.GaugeField(L, 64, 0)
    f.upload(U)
    f.hb_subsweep(0.5, 3, 5, 2, 1, 2)
    orc.hb_subsweep(U, L, 0.5, 3, 5, 2, 1, 2)
    assert np.max(np.abs(f.download() - U)) < 1e-12
