"""Imports, exports and copies between storage formats at the edges of the 32-half-site tiles: they move and
round values, so the results are equal, not close."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LATTICES = [(2, 2, 2, 2), (6, 2, 2, 4), (10, 6, 2, 2), (4, 4, 4, 4), (6, 6, 6, 6), (14, 10, 6, 2)]
FORMATS = [(64, 0), (64, 1), (32, 0), (32, 1)]


def stored(U, prec, store):
    """What a field of the format holds of U: the precision, and for 12 reals the first two rows."""
    W = U.astype(np.complex64).astype(np.complex128) if prec == 32 else U.copy()
    return W[..., :2, :] if store else W


@pytest.mark.parametrize("L", LATTICES)
@pytest.mark.parametrize("prec,store", FORMATS)
def test_import_and_export(gpu, orc, L, prec, store):
    U = orc.hot_start(L, 21)
    f = gpu.GaugeField(L, prec, store)
    f.upload(U)
    W = f.download()
    want = stored(U, prec, store)
    assert np.array_equal(W[..., : want.shape[-2], :], want)


@pytest.mark.parametrize("L", LATTICES)
@pytest.mark.parametrize("src", FORMATS)
@pytest.mark.parametrize("dst", FORMATS)
def test_copy_equals_export_and_import(gpu, orc, L, src, dst):
    f = gpu.GaugeField(L, *src)
    f.upload(orc.hot_start(L, 22))
    g = gpu.GaugeField(L, *dst)
    g.copy_from(f)
    h = gpu.GaugeField(L, *dst)
    h.upload(f.download())
    assert np.array_equal(g.download(), h.download())
