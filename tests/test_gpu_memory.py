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


class _Reserve:
    """All free device memory but `keep` bytes, held by another library."""

    def __init__(self, keep):
        import torch
        torch.cuda.empty_cache()
        self.t = torch.empty(torch.cuda.mem_get_info()[0] - keep, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        import torch
        self.t = None
        torch.cuda.empty_cache()


def test_kept_blocks_serve_other_contexts():
    """A field and its staging buffer fit although another context keeps what is missing."""
    import cl2qcd_b200 as c2q
    a, b = c2q.System(0), c2q.System(0)
    a.trim()  # nothing unused is left in the device's pool
    gfs = [c2q.Gaugefield(a, c2q.Lattice(24, 48)) for _ in range(3)]  # 382 MB each
    for gf in gfs:
        gf._destroy()
    L = c2q.Lattice(32, 64)  # 201 MB a field, as much staging
    with _Reserve(300 << 20):
        src = c2q.host.generate_source(L.seo, "z2", 80)
        f = c2q.Spinorfield_eo(b, L, src)
        assert np.array_equal(f.dump(), src)
        f._destroy()
    assert a.trim() == 0
    a.close()
    b.close()


def test_a_failed_buffer_leaves_none():
    """A staging buffer that found no memory: the call fails, a later smaller one works."""
    import cl2qcd_b200 as c2q
    s = c2q.System(0)
    L, l = c2q.Lattice(24, 48), c2q.Lattice(8, 8)  # a full field of 24^3x48: 127 MB
    small = c2q.host.generate_source(l.seo, "z2", 81)
    g = c2q.Spinorfield_eo(s, l, small)
    e, o = c2q.Spinorfield_eo(s, L), c2q.Spinorfield_eo(s, L)
    s.trim()  # nothing unused is left in the device's pool
    with _Reserve(64 << 20):
        with pytest.raises(c2q._lib.C2QError):
            c2q.host.convert_to_eoprec(e, o, np.zeros((L.vol, 24)))
        h = c2q.Spinorfield_eo(s, l, small)
        assert np.array_equal(h.dump(), g.dump())
    s.close()


def test_what_is_kept():
    """Blocks of a gauge field are kept unless another context has read it; trim gives them back."""
    import cl2qcd_b200 as c2q
    a, b = c2q.System(0), c2q.System(0)
    L = c2q.Lattice(8, 8)
    g = c2q.host.generate_gaugefield(L, 0.3, 82)
    src = c2q.host.generate_source(L.seo, "z2", 82)
    for prec in (64, 16):
        for reader in (a, b):
            gf = c2q.Gaugefield(a, L, g)
            out, inp = c2q.Spinorfield_eo(reader, L, precision=prec), c2q.Spinorfield_eo(reader, L, src, precision=prec)
            c2q.host.dslash(out, gf, inp, c2q.host.ODD, 0.15)
            n = a.lib.c2q_gauge_device_bytes(gf.h)
            gf._destroy()
            assert a.trim() == (n if reader is a else 0)
            assert a.trim() == 0 and b.trim() == 0
    b.close()
    a.close()


def test_server_keeps_no_scratch():
    """A registered gauge field takes the memory that the budget counts for it, and staging."""
    import torch
    import cl2qcd_b200 as c2q
    L = c2q.Lattice(16, 32)
    g = c2q.host.generate_gaugefield(L, 0.3, 83)  # 75 MB as uploaded
    server = c2q.host.Server(0, slots=1, precision=16)
    free = torch.cuda.mem_get_info()[0]
    server.add_gauge(1, L, g)
    used = free - torch.cuda.mem_get_info()[0]
    counted = server.stats()["gauge_bytes"]
    server.close()
    # staging of the upload, and each allocation in whole pages of 2 MiB
    assert used <= counted + g.nbytes + (32 << 20), (used, counted)
