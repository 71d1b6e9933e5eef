"""GPU: transfers of pageable and pinned host arrays (hostcopy.cu) around the chunk and
ring sizes (4 MiB chunks, a ring of four; below two chunks the plain copy): what comes
back is what went in, bit for bit."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


# bytes of a spinor field: 0.4 MB (plain), 8.0 MiB less a little, 8.96 MB (two chunks and a rest), 35 MB (the
# ring goes round, ragged end)
@pytest.mark.parametrize("ns,nt", [(8, 8), (14, 30), (18, 16), (22, 34)])
@pytest.mark.parametrize("pinned", [False, True])
def test_round_trip(system, ns, nt, pinned):
    import torch
    import cl2qcd_b200 as c2q
    L = c2q.Lattice(ns, nt)
    rng = np.random.default_rng(ns * 100 + nt)

    def host(shape):
        a = rng.standard_normal(shape)
        if pinned:
            t = torch.empty(shape, dtype=torch.float64, pin_memory=True)
            t.numpy()[...] = a
            return t.numpy()
        return a

    s = host((L.seo, 24))
    f = c2q.Spinorfield_eo(system, L, s)
    assert np.array_equal(f.dump(), s)
    full = host((L.vol, 24))
    e, o = c2q.Spinorfield_eo(system, L), c2q.Spinorfield_eo(system, L)
    c2q.host.convert_to_eoprec(e, o, full)
    assert np.array_equal(c2q.host.convert_from_eoprec(e, o), full)
    u = host((4 * L.vol, 18))
    assert np.array_equal(c2q.Gaugefield(system, L, u).download(), u)
    m = host((4 * L.vol, 8))
    assert np.array_equal(c2q.host.Gaugemomenta(system, L, m).download(), m)


@pytest.mark.parametrize("threads", [1, 3])
def test_omp_num_threads(lib, threads):
    """The copies take no more threads than OMP_NUM_THREADS allows (a launcher sets it to 1 where
    every GPU has its own process)."""
    code = """
import os, numpy as np, cl2qcd_b200 as c2q
s = c2q.System(0)
L = c2q.Lattice(18, 16)
f = c2q.Spinorfield_eo(s, L)
a = np.ones((L.seo, 24))
n = len(os.listdir("/proc/self/task"))
f.load(a)
assert np.array_equal(f.dump(), a)
print("new threads:", len(os.listdir("/proc/self/task")) - n)
"""
    env = dict(os.environ, OMP_NUM_THREADS=str(threads), PYTHONPATH=ROOT)
    out = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    assert int(out.stdout.split("new threads:")[1]) <= threads - 1
