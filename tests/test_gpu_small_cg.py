"""GPU: the cooperative CG iterations of small lattices (pcg.cuh, pcg64.cu) against the
per-launch iterations, which per-launch profiling selects, and the oracle's operator.

Lattices at the edges of the tiles (128 slots of two sites; 32 sites): one tile, a whole
number of tiles, a ragged last tile.  The mixed-precision iterations are the same
arithmetic in the same order: bitwise.  The FP64 ones differ by rounding: the same
iteration count, and solutions of two solves to the same residual."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

LATTICES = [(4, 4), (4, 8), (6, 12), (10, 8), (8, 16)]


def _solve(c2q, system, L, gf, srcs, params, add, action="twistedmass", per_launch=False):
    bs = [c2q.Spinorfield_eo(system, L, s) for s in srcs]
    xs = [c2q.Spinorfield_eo(system, L) for _ in srcs]
    reps = []
    system.lib.c2q_ctx_profile(system.h, int(per_launch))
    try:
        c2q.host.cg_multi(xs, c2q.host.QplusQminus_eo(action), gf, bs, params, add, reps)
    finally:
        system.lib.c2q_ctx_profile(system.h, 0)
    return [x.dump() for x in xs], reps


@pytest.mark.parametrize("ns,nt", LATTICES)
@pytest.mark.parametrize("precision,rec12,action", [(16, True, "twistedmass"), (16, False, "wilson"),
                                                    (32, True, "wilson"), (32, False, "twistedmass")])
@pytest.mark.parametrize("n", [1, 3])
def test_mixed_iterations_bitwise(port, system, O, ns, nt, precision, rec12, action, n):
    import cl2qcd_b200 as c2q
    port.set_lattice(ns, nt, 1.0, 0.0)
    L = c2q.Lattice(ns, nt, 1.0, 0.0)
    g = c2q.host.generate_gaugefield(L, 0.3, 11)
    gf = c2q.Gaugefield(system, L, g)
    srcs = [c2q.host.generate_source(L.seo, "z2" if k else "gaussian", 40 + k) for k in range(n)]
    kappa, mubar = (0.12, 0.0) if action == "wilson" else (0.14, 2 * 0.14 * 0.05)
    add = c2q.AdditionalParameters(kappa, mubar)
    P = c2q.SolverParameters(solver="cg", prec=0.0, rel_tol=1e-10, cgmax=5000, precision=precision, use_rec12=rec12)
    xa, ra = _solve(c2q, system, L, gf, srcs, P, add, action)
    xb, rb = _solve(c2q, system, L, gf, srcs, P, add, action, per_launch=True)
    for k in range(n):
        assert ra[k]["iterations"] == rb[k]["iterations"]
        assert ra[k]["reliable_updates"] == rb[k]["reliable_updates"]
        assert ra[k]["dslash_applications"] == rb[k]["dslash_applications"]
        assert np.array_equal(xa[k], xb[k])
        r = port.apply(O.OP_QPQM_EO, xa[k], g, kappa, mubar, action=O.WILSON if action == "wilson" else O.TWISTEDMASS)
        assert np.linalg.norm(r - srcs[k]) / np.linalg.norm(srcs[k]) <= 1.5e-10


def test_links_of_the_update_near_the_threshold(system):
    """The update's level and the threshold passed in one step: the update takes the links that the
    per-launch path takes.  Row 2 of the links is off by what still counts as SU(3), so that 12- and
    18-real residuals differ; at this kappa the residual rises between steps, so that some updates
    end above the threshold and the solve goes on from their residual.  Bitwise the same."""
    import cl2qcd_b200 as c2q
    L = c2q.Lattice(8, 8, 1.0, 0.0)
    g = c2q.host.generate_gaugefield(L, 0.3, 15).reshape(-1, 18).copy()
    g[:, 12:] += 4e-14 * np.random.default_rng(5).uniform(-1, 1, (len(g), 6))
    gf = c2q.Gaugefield(system, L, g)
    add = c2q.AdditionalParameters(0.25, 2 * 0.25 * 0.0005)
    src = c2q.host.generate_source(L.seo, "gaussian", 52)
    updates = set()
    for tol in np.geomspace(0.3, 1e-4, 200):
        # the update's level, counted from |r| = |b| at the start, lies just above the threshold
        P = c2q.SolverParameters(solver="cg", prec=0.0, rel_tol=tol, cgmax=20000, precision=16, use_rec12=True,
                                 reliable_delta=1.01 * tol)
        xa, ra = _solve(c2q, system, L, gf, [src], P, add)
        xb, rb = _solve(c2q, system, L, gf, [src], P, add, per_launch=True)
        assert ra[0]["iterations"] == rb[0]["iterations"]
        assert ra[0]["reliable_updates"] == rb[0]["reliable_updates"]
        assert np.array_equal(xa[0], xb[0]), tol
        updates.add(ra[0]["reliable_updates"])
    assert len(updates) > 1  # some solves did go on


@pytest.mark.parametrize("precision", [16, 32])
def test_batch_that_shrinks_into_one_launch(system, precision):
    """41 tiles a right-hand side, 12 of them: too many for one wave until some have converged
    (they start at solutions of different quality).  Bitwise the per-launch iterates."""
    import cl2qcd_b200 as c2q
    L = c2q.Lattice(12, 12, 1.0, 0.0)
    gf = c2q.Gaugefield(system, L, c2q.host.generate_gaugefield(L, 0.3, 14))
    add = c2q.AdditionalParameters(0.14, 2 * 0.14 * 0.05)
    A = c2q.host.QplusQminus_eo()

    def params(tol):
        return c2q.SolverParameters(solver="cg", prec=0.0, rel_tol=tol, cgmax=5000, precision=precision,
                                    use_rec12=True)

    bs = [c2q.Spinorfield_eo(system, L, c2q.host.generate_source(L.seo, "gaussian", 90 + k)) for k in range(12)]
    start = []
    for k, b in enumerate(bs):
        x = c2q.Spinorfield_eo(system, L)
        if k:
            c2q.host.cg(x, A, gf, b, params(10.0 ** (-0.75 * k)), add)
        start.append(x.dump())
    out = []
    for per_launch in (0, 1):
        xs = [c2q.Spinorfield_eo(system, L, s) for s in start]
        reps = []
        system.lib.c2q_ctx_profile(system.h, per_launch)
        try:
            c2q.host.cg_multi(xs, A, gf, bs, params(1e-10), add, reps)
        finally:
            system.lib.c2q_ctx_profile(system.h, 0)
        out.append(([x.dump() for x in xs], reps))
    its = [r["iterations"] for r in out[0][1]]
    assert len(set(its)) > 4 and max(r["true_resid_rel"] for r in out[0][1]) <= 1e-10
    for k in range(12):
        assert its[k] == out[1][1][k]["iterations"]
        assert out[0][1][k]["reliable_updates"] == out[1][1][k]["reliable_updates"]
        assert np.array_equal(out[0][0][k], out[1][0][k])


@pytest.mark.parametrize("ns,nt", LATTICES + [(6, 10)])
@pytest.mark.parametrize("rec12,action", [(False, "twistedmass"), (True, "wilson")])
@pytest.mark.parametrize("mode", ["rel_tol", "refresh", "prec"])
def test_fp64_iterations(port, system, O, ns, nt, rec12, action, mode):
    import cl2qcd_b200 as c2q
    port.set_lattice(ns, nt, 1.0, 0.0)
    L = c2q.Lattice(ns, nt, 1.0, 0.0)
    g = c2q.host.generate_gaugefield(L, 0.3, 12)
    gf = c2q.Gaugefield(system, L, g)
    src = c2q.host.generate_source(L.seo, "gaussian", 50)
    kappa, mubar = (0.12, 0.0) if action == "wilson" else (0.14, 2 * 0.14 * 0.05)
    add = c2q.AdditionalParameters(kappa, mubar)
    kw = {"rel_tol": dict(prec=0.0, rel_tol=1e-10), "refresh": dict(prec=0.0, rel_tol=1e-10, iter_refresh=7),
          "prec": dict(prec=1e-20 * float(np.sum(src ** 2)), resid_check_every=3)}[mode]
    P = c2q.SolverParameters(solver="cg", cgmax=5000, precision=64, use_rec12=rec12, **kw)
    xa, ra = _solve(c2q, system, L, gf, [src], P, add, action)
    xb, rb = _solve(c2q, system, L, gf, [src], P, add, action, per_launch=True)
    assert abs(ra[0]["iterations"] - rb[0]["iterations"]) <= (3 if mode == "prec" else 1)
    assert ra[0]["true_resid_rel"] <= 1e-10
    r = port.apply(O.OP_QPQM_EO, xa[0], g, kappa, mubar, action=O.WILSON if action == "wilson" else O.TWISTEDMASS)
    assert np.linalg.norm(r - src) / np.linalg.norm(src) <= 1.01e-10
    assert rel_l2(xa[0], xb[0]) <= 1e-8


@pytest.mark.parametrize("precision,mode", [(64, "rel_tol"), (64, "prec"), (64, "graph"), (32, "one"), (16, "one"),
                                            (16, "batch"), (16, "graph")])
def test_a_barrier_that_gives_up(port, O, precision, mode):
    """Barriers that one block too many is awaited at: the wait runs out, the launch is
    given up and the solve goes on without it.  The context works as before afterwards."""
    import cl2qcd_b200 as c2q
    system = c2q.System(0)
    port.set_lattice(8, 16, 1.0, 0.0)
    L = c2q.Lattice(8, 16, 1.0, 0.0)
    g = c2q.host.generate_gaugefield(L, 0.3, 16)
    gf = c2q.Gaugefield(system, L, g)
    kappa, mubar = 0.14, 2 * 0.14 * 0.05
    add = c2q.AdditionalParameters(kappa, mubar)
    srcs = [c2q.host.generate_source(L.seo, "gaussian", 53 + k) for k in range(5 if mode == "batch" else 1)]
    kw = dict(prec=1e-20 * float(np.sum(srcs[0] ** 2))) if mode == "prec" else dict(prec=0.0, rel_tol=1e-10)
    P = c2q.SolverParameters(solver="cg", cgmax=5000, precision=precision, use_rec12=True, use_graph=mode == "graph",
                             **kw)
    want, rep = _solve(c2q, system, L, gf, srcs, P, add)
    assert system.barrier_giveups == 0
    system.set_cooperative(2)
    xs, reps = _solve(c2q, system, L, gf, srcs, P, add)
    assert system.barrier_giveups == 1
    for k, s in enumerate(srcs):
        r = port.apply(O.OP_QPQM_EO, xs[k], g, kappa, mubar)
        assert np.linalg.norm(r - s) / np.linalg.norm(s) <= 1.5e-10
        # one iteration lost and the search direction begun anew; with prec a check interval of 10
        assert reps[k]["iterations"] <= rep[k]["iterations"] + 10
    system.set_cooperative(1)
    again, _ = _solve(c2q, system, L, gf, srcs, P, add)
    assert all(np.array_equal(a, w) for a, w in zip(again, want)) and system.barrier_giveups == 1
    system.close()


@pytest.mark.parametrize("precision", [64, 32, 16])
def test_more_iterations_than_a_launch_takes(system, precision):
    """Over a hundred iterations between two decisions: one launch after the other, nothing done to
    the solution in between."""
    import cl2qcd_b200 as c2q
    L = c2q.Lattice(12, 24, 1.0, 0.0)
    gf = c2q.Gaugefield(system, L, c2q.host.generate_gaugefield(L, 0.3, 51))
    add = c2q.AdditionalParameters(0.155, 2 * 0.155 * 1e-4)
    src = c2q.host.generate_source(L.seo, "gaussian", 64)
    tol = 1e-5
    P = c2q.SolverParameters(solver="cg", prec=0.0, rel_tol=tol, cgmax=5000, precision=precision, use_rec12=True,
                             iter_refresh=1000, reliable_delta=1e-9)
    xa, ra = _solve(c2q, system, L, gf, [src], P, add)
    xb, rb = _solve(c2q, system, L, gf, [src], P, add, per_launch=True)
    assert rb[0]["iterations"] > 110 and ra[0]["true_resid_rel"] <= tol
    if precision == 64:
        assert abs(ra[0]["iterations"] - rb[0]["iterations"]) <= 2
    else:
        for key in ("iterations", "reliable_updates", "dslash_applications"):
            assert ra[0][key] == rb[0][key], key
        assert np.array_equal(xa[0], xb[0])


@pytest.mark.parametrize("precision,n", [(16, 7), (16, 1), (64, 1)])
def test_solves_side_by_side(precision, n):
    """Cooperative grids of several contexts, that do not fit side by side with seven sources each
    (some iterations then run as ordinary launches, in between and with graphs): every solution is
    bitwise that of a solve with the device to itself."""
    import threading

    import cl2qcd_b200 as c2q
    L = c2q.Lattice(12, 12, 1.0, 0.0)  # 41 tiles: seven sources fill two thirds of the device
    g = c2q.host.generate_gaugefield(L, 0.3, 18)
    add = c2q.AdditionalParameters(0.15, 2 * 0.15 * 0.01)
    srcs = [c2q.host.generate_source(L.seo, "gaussian", 57 + k) for k in range(n)]

    def params(graph):
        return c2q.SolverParameters(solver="cg", prec=0.0, rel_tol=1e-10, cgmax=5000, precision=precision,
                                    use_rec12=True, use_graph=graph)

    alone = c2q.System(0)
    want, reps = _solve(c2q, alone, L, c2q.Gaugefield(alone, L, g), srcs, params(False), add)
    cooperative = alone.launch_count
    bad = []

    def work(i):
        try:
            s = c2q.System(0)
            gf = c2q.Gaugefield(s, L, g)
            for k in range(8):
                xs, r = _solve(c2q, s, L, gf, srcs, params(bool((i + k) % 2)), add)
                assert [q["iterations"] for q in r] == [q["iterations"] for q in reps]
                assert all(np.array_equal(a, b) for a, b in zip(xs, want))
            launches[i] = s.launch_count
            s.close()
        except Exception as e:
            bad.append(e)

    launches = [0] * 4
    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad
    # (both kinds of iteration were met: a cooperative solve has few launches)
    assert n < 7 or max(launches) > 8 * cooperative
    alone.close()


@pytest.mark.parametrize("choice,n", [(0, 1), (3, 1), (4, 3)])
def test_a_pinned_sweep_choice_is_run(system, choice, n):
    """While a choice is pinned the sweeps are launches of their own, with that choice: at least the
    four of an iteration and its p update, and bitwise the cooperative launch's solutions."""
    import cl2qcd_b200 as c2q
    L = c2q.Lattice(6, 12, 1.0, 0.0)
    gf = c2q.Gaugefield(system, L, c2q.host.generate_gaugefield(L, 0.3, 17))
    add = c2q.AdditionalParameters(0.14, 2 * 0.14 * 0.05)
    srcs = [c2q.host.generate_source(L.seo, "gaussian", 56 + k) for k in range(n)]
    P = c2q.SolverParameters(solver="cg", prec=0.0, rel_tol=1e-10, cgmax=5000, precision=16, use_rec12=True)
    want, rep = _solve(c2q, system, L, gf, srcs, P, add)
    system.set_sweep_choice(choice)
    try:
        before = system.launch_count
        xs, reps = _solve(c2q, system, L, gf, srcs, P, add)
        launches = system.launch_count - before
    finally:
        system.set_sweep_choice(-1)
    assert launches >= 5 * max(r["iterations"] for r in reps)
    assert all(np.array_equal(a, b) for a, b in zip(xs, want))


@pytest.mark.parametrize("precision", [64, 32, 16])
def test_limits_and_nan(system, precision):
    """The iteration limit and a residual that is no number end the solve as before."""
    import cl2qcd_b200 as c2q
    L = c2q.Lattice(6, 8, 1.0, 0.0)
    gf = c2q.Gaugefield(system, L, c2q.host.generate_gaugefield(L, 0.3, 13))
    add = c2q.AdditionalParameters(0.14, 2 * 0.14 * 0.05)
    src = c2q.host.generate_source(L.seo, "z2", 51)
    for cgmax in (1, 2, 9):
        x, b = c2q.Spinorfield_eo(system, L), c2q.Spinorfield_eo(system, L, src)
        rep = {}
        with pytest.raises(c2q.SolverDidNotSolve):
            c2q.host.cg(x, c2q.host.QplusQminus_eo(), gf, b,
                        c2q.SolverParameters(solver="cg", prec=0.0, rel_tol=1e-10, cgmax=cgmax, precision=precision),
                        add, rep)
        assert rep["iterations"] == cgmax and np.isfinite(rep["true_resid_rel"])
    src[3, 5] = np.nan
    x, b = c2q.Spinorfield_eo(system, L), c2q.Spinorfield_eo(system, L, src)
    with pytest.raises(c2q.SolverStuck) as stuck:
        c2q.host.cg(x, c2q.host.QplusQminus_eo(), gf, b,
                    c2q.SolverParameters(solver="cg", prec=0.0, rel_tol=1e-10, cgmax=50, precision=precision), add)
    assert stuck.value.iterations <= 2
