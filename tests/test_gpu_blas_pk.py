"""GPU: level-1 BLAS and conversions of the FP32 / FP16 slot fields (blas_pk.cuh) against numpy
in FP64 on the fields' own (rounded) values, on lattices whose slots fill part of a
block, exactly one, and several with a ragged last one; and gauge objects on reused
memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LATTICES = [(4, 4), (4, 8), (6, 12), (10, 12)]  # 64, 128, 648, 3000 slots


def _cplx(a):
    return a[:, 0::2] + 1j * a[:, 1::2]


def _error(got, ref, prec):
    """Largest deviation per site in units of the site's largest |component|."""
    scale = np.maximum(np.abs(ref.real), np.abs(ref.imag)).max(axis=1, keepdims=True)
    scale = np.where(scale > 0, scale, 1)
    d = got - ref
    return float((np.maximum(np.abs(d.real), np.abs(d.imag)) / scale).max())


# FP32: at most 8 roundings of 2^-24 on sums of up to 5 terms no larger than a few times the
# result's site scale; FP16 stores to half a step of 1 / 32767 of the site's scale
TOL = {32: 64 * 2.0 ** -24, 16: 0.51 / 32767 + 64 * 2.0 ** -24}


@pytest.mark.parametrize("ns,nt", LATTICES)
@pytest.mark.parametrize("prec", [32, 16])
def test_blas_on_slots(system, ns, nt, prec):
    import cl2qcd_b200 as c2q
    H = c2q.host
    L = c2q.Lattice(ns, nt)
    src = [H.generate_source(L.seo, "gaussian", 7 + k) for k in range(3)]
    f = [c2q.Spinorfield_eo(system, L, s, precision=prec) for s in src]
    x, y, z = (_cplx(g.dump()) for g in f)
    for v, s in zip((x, y, z), src):  # the upload's rounding
        assert _error(v, _cplx(s), prec) <= TOL[prec]
    out = c2q.Spinorfield_eo(system, L, precision=prec)
    a, b = 0.7 - 0.3j, -0.4 + 0.9j
    g5 = np.where(np.arange(12) < 6, 1, -1)

    def check(ref):
        assert _error(_cplx(out.dump()), ref, prec) <= TOL[prec]

    H.saxpy(out, a, f[0], f[1])
    check(y - a * x)
    H.saxpy_AND_gamma5_eo(out, a, f[0], f[1])
    check(g5 * (y - a * x))
    H.sax(out, a, f[0])
    check(a * x)
    H.saxsbypz(out, a, f[0], b, f[1], f[2])
    check(a * x + b * y + z)
    H.copyData(out, f[0])
    assert np.array_equal(out.dump(), f[0].dump())
    out.gamma5()
    check(g5 * x)
    H.M_tm_sitediagonal(out, f[0], 0.3)
    check((1 + 0.3j * g5) * x)
    # reductions: FP32 products, FP64 sums
    n = np.linalg.norm(x) * np.linalg.norm(y)
    assert abs(H.scalar_product(f[0], f[1]) - np.vdot(x, y)) <= 1e-6 * n
    assert abs(H.squarenorm(f[0]) - np.linalg.norm(x) ** 2) <= 1e-6 * np.linalg.norm(x) ** 2
    r = H.saxpy_AND_squarenorm(out, a, f[0], f[1])
    assert abs(r - np.linalg.norm(y - a * x) ** 2) <= 1e-6 * np.linalg.norm(y - a * x) ** 2
    # conversions between the slot precisions and FP64
    for p in (64, 32, 16):
        o = c2q.Spinorfield_eo(system, L, precision=p)
        o.convert_from(f[0])
        assert _error(_cplx(o.dump()), x, p) <= (TOL[p] if p != 64 else 0.0)


def test_gauge_objects_on_reused_memory(system):
    """A gauge field created on another's freed blocks: operators and derived copies are its own."""
    import cl2qcd_b200 as c2q
    H = c2q.host
    add = c2q.AdditionalParameters(0.14, 2 * 0.14 * 0.05)
    P = c2q.SolverParameters(solver="cg", prec=0.0, rel_tol=1e-10, cgmax=5000, precision=16, use_rec12=True)

    def solve(sysm, L, seed):
        gf = c2q.Gaugefield(sysm, L, H.generate_gaugefield(L, 0.3, seed))
        b = c2q.Spinorfield_eo(sysm, L, H.generate_source(L.seo, "z2", seed))
        x = c2q.Spinorfield_eo(sysm, L)
        H.cg(x, H.QplusQminus_eo(), gf, b, P, add)
        return x.dump()

    lats = [c2q.Lattice(6, 8, 1.0, 0.0), c2q.Lattice(4, 8, 1.0, 0.0), c2q.Lattice(6, 8, 1.0, 0.0)]
    here = [solve(system, L, 30 + k) for k, L in enumerate(lats)]
    for k, L in enumerate(lats):
        fresh = c2q.System(0)
        assert np.array_equal(here[k], solve(fresh, L, 30 + k))
        fresh.close()
