"""Copies into a field whose prefetched configuration waits for its commit: refused from another format, as
qcb.h states, and done within the format."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = (6, 4, 4, 2)


@pytest.mark.parametrize("src", [(64, 0), (64, 1), (32, 0), (32, 1)])
def test_copy_while_a_prefetch_waits(gpu, orc, src):
    U = orc.hot_start(L, 1)
    f, g = gpu.GaugeField(L, 64, 0), gpu.GaugeField(L, *src)
    f.hot_start(5)
    g.hot_start(6)
    held, links = f.download(), g.download()
    f.prefetch(U)
    if src == (64, 0):
        f.copy_from(g)
        want = links
    else:
        with pytest.raises(gpu.QcbError) as e:
            f.copy_from(g)
        assert e.value.code == -1
        want = held
    h = gpu.GaugeField(L, 64, 0)
    h.copy_from(f)  # the links themselves, past the staging buffer
    assert np.array_equal(h.download(), want)
    f.commit_prefetch()
    assert np.array_equal(f.download(), U)
