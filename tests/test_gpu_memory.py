"""GPU: memory of gauge objects (link_alloc in fields.cu): freed blocks kept for the next
object of the same size, beside stream captures of other threads, for fields that several
contexts read, and given back when memory is asked for elsewhere."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _in_thread(f):
    err = []

    def run():
        try:
            f()
        except Exception as e:  # handed to the test's thread
            err.append(e)
    t = threading.Thread(target=run)
    t.start()
    t.join()
    if err:
        raise err[0]


@pytest.mark.parametrize("derived", [False, True])
def test_destroy_beside_a_capture(system, derived):
    """Gauge objects go while another thread captures a stream: the capture stays valid, and
    memory that is used again holds its new owner's links."""
    import torch
    import cl2qcd_b200 as c2q
    L = c2q.Lattice(4, 8)
    gs = [c2q.host.generate_gaugefield(L, 0.3, 60 + k) for k in range(3)]
    src = c2q.host.generate_source(L.seo, "gaussian", 61)
    out = c2q.Spinorfield_eo(system, L, precision=32 if derived else 64)
    inp = c2q.Spinorfield_eo(system, L, src, precision=32 if derived else 64)

    def hop(gf):
        c2q.host.dslash(out, gf, inp, c2q.host.ODD, 0.15)
        return out.dump()

    want = []
    for g in gs:
        gf = c2q.Gaugefield(system, L, g)
        want.append(hop(gf))
        del gf
    t = torch.arange(1024, dtype=torch.float32, device="cuda")
    r = torch.zeros_like(t)
    torch.cuda.synchronize()
    old, mom = c2q.Gaugefield(system, L, gs[0]), c2q.host.Gaugemomenta(system, L)
    assert np.array_equal(hop(old), want[0])
    graph = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        graph.capture_begin(capture_error_mode="thread_local")
        torch.mul(t, 2, out=r)
        _in_thread(lambda: (old._destroy(), mom._destroy()))
        graph.capture_end()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(r, 2 * t)
    for g, w in zip(gs[1:], want[1:]):
        gf = c2q.Gaugefield(system, L, g)
        assert np.array_equal(hop(gf), w)


def test_contexts_in_threads():
    """Each context in a thread of its own, gauge objects coming and going."""
    import cl2qcd_b200 as c2q
    lats = [c2q.Lattice(4, 4), c2q.Lattice(4, 8)]
    gs = [c2q.host.generate_gaugefield(L, 0.3, 70) for L in lats]

    def work():
        s = c2q.System(0)
        for k in range(40):
            L, g = lats[k % 2], gs[k % 2]
            gf, m = c2q.Gaugefield(s, L, g), c2q.host.Gaugemomenta(s, L)
            if k % 5 == 0:
                assert np.array_equal(gf.download(), g)
            gf._destroy()
            m._destroy()
        s.close()

    err = []

    def run():
        try:
            work()
        except Exception as e:
            err.append(e)
    ts = [threading.Thread(target=run) for _ in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not err, err
