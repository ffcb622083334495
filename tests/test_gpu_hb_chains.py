"""Single chains side by side on their own streams, and the small lattices' heatbath kernel at its line.

A chain alone does not fill the GPU, so eight of them in one CUDA graph overlap.  A kernel that gains on one
chain by taking the SMs of the others would show here.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chains(gpu, L, n):
    out = []
    for i in range(n):
        f = gpu.GaugeField(L, 64, 0)
        f.hot_start(i + 1)
        f.sync()
        out.append(f)
    return out


def captured(torch, fields, sweeps):
    """A graph of the fields' sweeps, each field on a stream of its own, forked from and joined to one."""
    root, own = torch.cuda.Stream(), [torch.cuda.Stream() for _ in fields]
    for f, s in zip(fields, own):
        f.set_stream(s.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=root):
        fork = torch.cuda.Event()
        fork.record(root)
        for s in own:
            s.wait_event(fork)
        for k in range(sweeps):
            for f in fields:
                f.hb_sweep(6.0, 2, 5, k)
        for s in own:
            join = torch.cuda.Event()
            join.record(s)
            root.wait_event(join)
    return graph, root


def seconds(torch, graph, root):
    a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    best = 1e9
    for _ in range(6):
        torch.cuda.synchronize()
        with torch.cuda.stream(root):
            a.record(root)
            for _ in range(4):
                graph.replay()
            b.record(root)
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 1e-3)
    return best


@pytest.mark.parametrize("L", [(12, 12, 12, 8), (10, 10, 10, 10)])
def test_eight_chains_overlap(gpu, L):
    """A set of these lattices is 216 and 157 warps of links, eight of them three and two a scheduler, each mostly
    waiting for its own chain: less than three times one chain's time (1.5 and 1.3 times with one lane a link; it
    was seven and six times with eight)."""
    torch = pytest.importorskip("torch")
    t = []
    for n in (1, 8):
        fields = chains(gpu, L, n)
        graph, root = captured(torch, fields, 6)
        t.append(seconds(torch, graph, root))
        del graph
        torch.cuda.synchronize()
        for f in fields:
            f.close()
    assert t[1] < 3.0 * t[0], t


@pytest.mark.parametrize("L", [(4, 4, 4, 4), (8, 8, 8, 8), (12, 12, 12, 8)])
def test_captured_chains_equal_single_ones(gpu, L):
    torch = pytest.importorskip("torch")
    side, alone = chains(gpu, L, 3), chains(gpu, L, 3)
    graph, root = captured(torch, side, 2)
    with torch.cuda.stream(root):
        graph.replay()
        graph.replay()
    torch.cuda.synchronize()
    for f, g in zip(side, alone):
        for _ in range(2):
            for k in range(2):
                g.hb_sweep(6.0, 2, 5, k)
        assert np.array_equal(f.download(), g.download())
    del graph
    torch.cuda.synchronize()


# 2304, 2368 (the line between the kernels) and 2560 half-sites
@pytest.mark.parametrize("L", [(12, 8, 8, 6), (74, 4, 4, 4), (8, 8, 8, 10)])
@pytest.mark.parametrize("store", [0, 1])
@pytest.mark.parametrize("n_hits", [0, 1, 2, 3, 5])
def test_sweeps_at_the_line_equal_the_batch(gpu, L, store, n_hits):
    """The one-thread kernel of a one-chain batch draws from the same streams: equal links.  Three hits and more
    fill the table of draws again; a coupling of 2 makes links run past it."""
    for beta in (5.9, 2.0):
        f = gpu.GaugeField(L, 64, store)
        f.hot_start(11)
        b = gpu.Batch([L], [beta], [77], 64, store)
        b.upload(0, f.download())
        f.upload(f.download())
        for sweep in range(2):
            f.hb_sweep(beta, n_hits, 77, sweep)
        b.sweep(n_hits, 2)
        b.sync()
        assert np.array_equal(f.download(), b.download(0))
