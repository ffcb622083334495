"""The server's copies of request links: rounded to its format by several threads, in buffers that later
requests use again.  Different configurations one after the other and from several threads at once, against the
measured flow of a field with the same links."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# a lattice smaller than a tile, one whose input four threads share, one that runs alone (2^17 half-sites)
LATTICES = [(6, 2, 2, 2), (12, 12, 12, 8), (16, 16, 16, 64)]


def measured(gpu, L, U, prec, store, n):
    f = gpu.GaugeField(L, 64, 0)
    f.upload(U)
    fl = gpu.GradientFlow(f, 0.02, prec=prec, store=store)
    return fl.measure(f, n, 1)


def links(gpu, L, seed):
    f = gpu.GaugeField(L, 64, 0)
    f.hot_start(seed)
    return f.download()


@pytest.mark.parametrize("prec,store", [(64, 0), (64, 1), (32, 0), (32, 1)])
def test_requests_one_after_another_and_together(gpu, prec, store):
    """Requests that run alone equal the measured flow bit for bit; those in shared launches sum their sites
    in another order, 1e-10 as in the serving tests."""
    srv = gpu.Server(8 << 30, prec=prec, store=store)
    inputs = {(i, seed): links(gpu, L, seed) for i, L in enumerate(LATTICES) for seed in (1, 2)}
    want = {k: measured(gpu, LATTICES[k[0]], U, prec, store, 3) for k, U in inputs.items()}

    def check(n):
        srv.wait(120.0)
        seen = 0
        while (r := srv.poll()) is not None:
            i, seed = r[0] % 10, r[0] // 10
            ref = want[i, seed]
            if i == 2:
                assert np.array_equal(r[1], ref), (i, seed)
            else:
                assert np.max(np.abs(r[1] - ref)) < 1e-10 * max(1.0, float(np.max(np.abs(ref)))), (i, seed)
            seen += 1
        assert seen == n

    for seed in (1, 2, 1):  # the same sizes again: the buffers of the requests before
        for i, L in enumerate(LATTICES):
            srv.submit(10 * seed + i, L, inputs[i, seed], 0.02, 3)
        check(len(LATTICES))
    keys = list(inputs)
    th = [threading.Thread(target=lambda k=k: srv.submit(10 * k[1] + k[0], LATTICES[k[0]], inputs[k], 0.02, 3))
          for k in keys]
    for t in th:
        t.start()
    for t in th:
        t.join()
    check(len(keys))
    srv.close()
