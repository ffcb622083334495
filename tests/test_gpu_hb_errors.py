"""Heatbath errors reach the host: a zero link has no SU(2) projection, which every update kernel flags and
skips.  A lattice of the small lattices' kernel and one past it, both precisions and storages, the single link,
and a batch.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ERANGE = -7
LATTICES = [(4, 4, 4, 4), (16, 12, 12, 8)]  # 128 and 9216 half-sites


def zeros(L):
    return np.zeros((int(np.prod(L)), 4, 3, 3), complex)


def raises_range(gpu, call):
    with pytest.raises(gpu.QcbError) as e:
        call()
    assert e.value.code == ERANGE and "projection" in str(e.value)


@pytest.mark.parametrize("L", LATTICES)
@pytest.mark.parametrize("prec,store", [(64, 0), (64, 1), (32, 0), (32, 1)])
def test_zero_links_raise_once(gpu, L, prec, store):
    f = gpu.GaugeField(L, prec, store)
    f.upload(zeros(L))
    f.plaquette()  # no update yet, no error
    f.hb_subsweep(6.0, 2, 1, 0, 1, 2)
    f.clover_qe()  # reads the results and leaves the flags
    raises_range(gpu, f.plaquette)
    f.plaquette()  # reported once
    if (prec, store) == (64, 0):
        assert not np.any(f.download())  # the links are left as they were
    f.hb_sweep(6.0, 0, 1, 0)
    f.plaquette()  # no hits, nothing to flag


@pytest.mark.parametrize("L", LATTICES)
def test_one_bad_link_among_good_ones(gpu, L):
    """The set's last link zero (w = u A = 0) raises; without it the sub-sweep raises nothing."""
    f = gpu.GaugeField(L, 64, 0)
    f.hot_start(3)
    U = f.download()
    f.hb_subsweep(6.0, 1, 1, 0, 0, 0)
    f.plaquette()
    V = U.copy()
    x = np.arange(len(U))
    c = [x // int(np.prod(L[:d])) % L[d] for d in range(4)]
    site = int(x[(sum(c) % 2) == 0][-1])
    V[site, 0] = 0.0
    f.upload(V)
    f.hb_subsweep(6.0, 1, 1, 0, 0, 0)
    raises_range(gpu, f.plaquette)
    assert not np.any(f.download()[site, 0])


def test_single_link_and_batch(gpu):
    L = (4, 4, 4, 4)
    f = gpu.GaugeField(L, 64, 0)
    f.upload(zeros(L))
    raises_range(gpu, lambda: f.hb_link(5, 1, 6.0, 1, 1, 0))
    f.plaquette()
    b = gpu.Batch([L, (8, 4, 4, 4)], [6.0, 6.0], [1, 2])
    b.hot_start()
    b.sweep(1, 1)
    b.sync()
    b.upload(1, zeros((8, 4, 4, 4)))
    b.sweep(1, 1)
    raises_range(gpu, b.sync)
    b.sync()
