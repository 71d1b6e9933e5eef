"""What a program built on this framework spends its time on, as cases that can be timed.

A case is one call (or one short sequence of calls) of the public Python surface
(``cl2qcd_b200.host``) on one lattice: an inversion with one of the solvers, a batch of
inversions, a repeated operator application, a fermion force, a burst of serving requests.
``prepare`` makes the gauge field and the sources a program has at hand, ``run`` is the call
with its results in pinned host memory, ``exact`` the same results from plain torch in
64 bits.
"""
import math

import numpy as np
import torch

from cl2qcd_b200 import host as c2q

REL_TOL = 1e-10  # every solve runs to this true residual
CHUNK = 1 << 22  # links made at a time


# ---------------------------------------------------------------- the cases
def listed():
    """Antiperiodic time, periodic space; eps is the disorder of the gauge field exp(i eps H)."""
    return [
        # the smallest inversions (tests, tuning of a physics point): latency and launches count
        dict(name="cg64 8^3x8 graph", kind="cg", ns=8, nt=8, eps=0.3, kappa=0.15, mu=0.01, precision=64,
             rec12=False, graph=True, nsrc=1, source="z2"),
        # the reference's own arithmetic at an ordinary size
        dict(name="cg64 24^3x48", kind="cg", ns=24, nt=48, eps=0.25, kappa=0.16, mu=0.005, precision=64,
             rec12=False, graph=False, nsrc=1, source="gaussian"),
        # mixed-precision inversions: a small volume, a ragged one in FP32, the production size, the largest
        dict(name="cg16 16^3x32", kind="cg", ns=16, nt=32, eps=0.3, kappa=0.15, mu=0.01, precision=16,
             rec12=True, graph=False, nsrc=1, source="z2"),
        dict(name="cg32 22^3x36", kind="cg", ns=22, nt=36, eps=0.25, kappa=0.15, mu=0.008, precision=32,
             rec12=False, graph=False, nsrc=1, source="gaussian"),
        dict(name="cg16 32^3x64", kind="cg", ns=32, nt=64, eps=0.25, kappa=0.16, mu=0.005, precision=16,
             rec12=True, graph=False, nsrc=1, source="gaussian"),
        dict(name="cg16 48^3x96", kind="cg", ns=48, nt=96, eps=0.2, kappa=0.1625, mu=0.003, precision=16,
             rec12=True, graph=False, nsrc=1, source="gaussian"),
        # the 12 point sources of a propagator, solved as one batch
        dict(name="cg16 24^3x48 12 sources", kind="cg", ns=24, nt=48, eps=0.25, kappa=0.16, mu=0.005, precision=16,
             rec12=True, graph=True, nsrc=12, source="point"),
        # BiCGStab on the Schur complement, where it converges (light hopping parameter)
        dict(name="bicgstab64 24^3x48", kind="bicgstab", ns=24, nt=48, eps=0.25, kappa=0.12, mu=0.005, precision=64,
             rec12=False, source="gaussian"),
        # a whole inversion of a host source field, result on the host (inverter programs)
        dict(name="inversion 20^3x40", kind="inversion", ns=20, nt=40, eps=0.25, kappa=0.12, mu=0.005,
             precision=64, rec12=False, solver="bicgstab"),
        # molecular dynamics: one fermion force, its solve included
        dict(name="force 16^3x32", kind="force", ns=16, nt=32, eps=0.25, kappa=0.15, mu=0.01, precision=16,
             rec12=True),
        # power iteration for the largest eigenvalue of Q+Q-: operator, BLAS and reductions
        dict(name="power64 32^3x64", kind="power", ns=32, nt=64, eps=0.25, kappa=0.16, mu=0.005, precision=64,
             rec12=False, count=12),
        # a burst of requests of two volumes to the server
        dict(name="serving 16^3x32 + 20^3x40", kind="serving", ns=16, nt=32, eps=0.25, kappa=0.15, mu=0.01,
             requests=6, nsrc=3),
    ]


def draw(rng):
    kind = rng.choice(["cg", "cg", "cg", "cg", "bicgstab", "inversion", "force", "power", "serving"])
    most = {"cg": 1 << 20, "bicgstab": 1 << 19, "inversion": 1 << 18, "force": 1 << 17, "power": 1 << 20,
            "serving": 1 << 16}[kind]
    c = dict(kind=kind, precision=rng.choice([64, 32, 16]), eps=round(rng.uniform(0.2, 0.35), 3),
             mu=round(math.exp(rng.uniform(math.log(0.008), math.log(0.02))), 5))
    c["kappa"] = round(rng.uniform(0.14, 0.16) if kind in ("cg", "force", "power", "serving")
                       else rng.uniform(0.11, 0.125), 4)
    if kind in ("cg", "power") and c["precision"] == 64:
        most >>= 1
    while True:
        # extents are even; the reduced precisions (and so the server) pair t and t + NT/2
        step = 2 if c["precision"] == 64 and kind != "serving" else 4
        c["ns"] = 2 * round(math.exp(rng.uniform(math.log(3), math.log(16))))
        c["nt"] = step * round(math.exp(rng.uniform(math.log(8 / step), math.log(64 / step))))
        if c["ns"] ** 3 * c["nt"] // 2 <= most:
            break
    c["rec12"] = rng.random() < 0.6 if c["precision"] != 64 else rng.random() < 0.2
    seo = c["ns"] ** 3 * c["nt"] // 2
    if kind == "cg":
        c["source"] = rng.choice(["z2", "gaussian", "point"])
        c["nsrc"] = min(rng.randint(1, 12), max(1, (1 << 21) // seo)) if rng.random() < 0.4 else 1
        if c["precision"] == 64:
            c["nsrc"] = min(c["nsrc"], 3)
        c["graph"] = rng.random() < 0.4
    elif kind == "bicgstab":
        c["source"] = rng.choice(["z2", "gaussian"])
    elif kind == "inversion":
        c["solver"] = rng.choice(["bicgstab", "bicgstab_save"])
    elif kind == "power":
        c["count"] = rng.randint(8, 24)
    elif kind == "serving":
        del c["precision"], c["rec12"]
        c["requests"], c["nsrc"] = rng.randint(3, 8), rng.randint(1, 6)
    return c


# ---------------------------------------------------------------- inputs
def _gen(seed, what):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + what) % (1 << 62))
    return g


def _mm(a, b):
    """3x3 complex products, matrices as lists of 9 component vectors."""
    return [sum(a[3 * r + k] * b[3 * k + c] for k in range(3)) for r in range(3) for c in range(3)]


def _links(ns, nt, eps, seed):
    """U = exp(i eps H), H traceless Hermitian with normal entries, as (4 V, 9) complex128 on the GPU."""
    n = 4 * ns ** 3 * nt
    out = torch.empty((n, 9), dtype=torch.complex128, device="cuda")
    gen = _gen(seed, 1)
    for at in range(0, n, CHUNK):
        m = min(CHUNK, n - at)
        z = torch.randn((9, m), dtype=torch.float64, device="cuda", generator=gen)
        tr = (z[0] + z[1] + z[2]) / 3
        lo = [torch.complex(z[3 + 2 * k], z[4 + 2 * k]) * math.sqrt(0.5) for k in range(3)]
        d = [torch.complex(z[k] - tr, torch.zeros_like(tr)) for k in range(3)]
        h = [d[0], lo[0], lo[1], lo[0].conj(), d[1], lo[2], lo[1].conj(), lo[2].conj(), d[2]]
        x = [1j * (eps / 4) * v for v in h]
        one = torch.ones(m, dtype=torch.complex128, device="cuda")
        u = [one * (k % 4 == 0) for k in range(9)]
        for k in range(10, 0, -1):  # Taylor by Horner, then two squarings
            u = [v / k for v in _mm(x, u)]
            for j in (0, 4, 8):
                u[j] = u[j] + 1
        for _ in range(2):
            u = _mm(u, u)
        # rows 0 and 1 orthonormal, row 2 their cross product
        r0, r1 = u[0:3], u[3:6]
        n0 = torch.sqrt(sum(v.abs() ** 2 for v in r0))
        r0 = [v / n0 for v in r0]
        ov = sum(a.conj() * b for a, b in zip(r0, r1))
        r1 = [b - ov * a for a, b in zip(r0, r1)]
        n1 = torch.sqrt(sum(v.abs() ** 2 for v in r1))
        r1 = [v / n1 for v in r1]
        r2 = [(r0[(k + 1) % 3] * r1[(k + 2) % 3] - r0[(k + 2) % 3] * r1[(k + 1) % 3]).conj() for k in range(3)]
        out[at:at + m] = torch.stack(r0 + r1 + r2, dim=1)
    return out


def _source(kind, n, seed, k=0):
    """One source field as (n, 24) float64 on the GPU."""
    if kind == "point":  # spin k % 4, colour k // 4, at a site of the seed's choice
        b = torch.zeros((n, 24), dtype=torch.float64, device="cuda")
        b[int(seed) * 7919 % n, 2 * (3 * (k % 4) + k // 4)] = 1.0
        return b
    gen = _gen(seed, 100 + k)
    if kind == "z2":
        return (torch.randint(0, 2, (n, 24), device="cuda", generator=gen).double() * 2 - 1) * math.sqrt(0.5)
    return torch.randn((n, 24), dtype=torch.float64, device="cuda", generator=gen)


_keep = {}


def _system():
    """One context for the life of the process, as a program keeps it."""
    if "system" not in _keep:
        _keep["system"] = c2q.System(0)
    return _keep["system"]


def _server():
    if "server" not in _keep:
        _keep["server"] = c2q.Server(0, slots=4, precision=16, rec12=True)
        _keep["gauges"] = 0
    return _keep["server"]


def _host_links(ns, nt, eps, seed):
    u = torch.view_as_real(_links(ns, nt, eps, seed)).reshape(-1)
    h = torch.empty(u.shape, dtype=torch.float64, pin_memory=True)
    h.copy_(u)
    return h.numpy()


def _lattice(ns, nt):
    return c2q.Lattice(ns, nt, theta_t=1.0)


def _params(case, solver):
    return c2q.SolverParameters(solver=solver, prec=0.0, rel_tol=REL_TOL, cgmax=40000,
                                precision=case["precision"], use_rec12=case["rec12"],
                                use_graph=case.get("graph", False))


def _field(system, lat, t):
    h = torch.empty(t.shape, dtype=torch.float64, pin_memory=True)
    h.copy_(t)
    return c2q.Spinorfield_eo(system, lat, h.numpy())


def _pinned(lat, n=1):
    return [torch.empty((lat.seo, 24), dtype=torch.float64, pin_memory=True) for _ in range(n)]


def _requests(case, seed):
    """(lattice number, kappa, mu, sources, source seed) of a burst."""
    got = []
    for k in range(case["requests"]):
        n = 1 + 5 * k % case["nsrc"]
        got.append((k % 2, case["kappa"] - 0.002 * (k % 3), case["mu"] * (1 + 0.25 * (k % 4)), n,
                    (int(seed) * 65537 + 1000 * k) % (1 << 40)))
    return got


def _two_lattices(case):
    return [_lattice(case["ns"], case["nt"]), _lattice(case["ns"] + 4, case["nt"] + 8)]


def prepare(case, seed):
    lat = _lattice(case["ns"], case["nt"])
    kind = case["kind"]
    st = {"case": case, "lat": lat}
    if kind == "serving":
        srv = _server()
        st["server"], st["gauges"] = srv, []
        for i, la in enumerate(_two_lattices(case)):
            _keep["gauges"] += 1
            srv.add_gauge(_keep["gauges"], la, _host_links(la.ns, la.nt, case["eps"], seed + 7 * i))
            st["gauges"].append((_keep["gauges"], la))
        st["requests"] = _requests(case, seed)
        st["out"] = [np.zeros((r[3], st["gauges"][r[0]][1].seo, 24)) for r in st["requests"]]
        return st
    system = st["system"] = _system()
    st["gf"] = c2q.Gaugefield(system, lat, _host_links(lat.ns, lat.nt, case["eps"], seed))
    st["add"] = c2q.AdditionalParameters.from_mu(case["kappa"], case["mu"])
    if kind == "cg":
        st["b"] = [_field(system, lat, _source(case["source"], lat.seo, seed, k)) for k in range(case["nsrc"])]
        st["x"] = [c2q.Spinorfield_eo(system, lat) for _ in range(case["nsrc"])]
        st["out"] = _pinned(lat, case["nsrc"])
        st["params"] = _params(case, "cg")
        st["A"] = c2q.QplusQminus_eo()
    elif kind == "bicgstab":
        st["b"] = [_field(system, lat, _source(case["source"], lat.seo, seed))]
        st["x"] = [c2q.Spinorfield_eo(system, lat)]
        st["out"] = _pinned(lat)
        st["params"] = _params(case, "bicgstab")
        st["A"] = c2q.Aee()
    elif kind == "inversion":
        st["source"] = _source("gaussian", lat.vol, seed).cpu().numpy()
        st["params"] = _params(case, case["solver"])
    elif kind == "force":
        st["phi"] = _field(system, lat, _source("gaussian", lat.seo, seed))
        st["gm"] = c2q.Gaugemomenta(system, lat)
        st["params"] = _params(case, "cg")
    elif kind == "power":
        st["start"] = c2q.Spinorfield_eo(system, lat, precision=case["precision"])
        st["full"] = _field(system, lat, _source("gaussian", lat.seo, seed))
        st["start"].convert_from(st["full"])
        st["x"] = [c2q.Spinorfield_eo(system, lat, precision=case["precision"]) for _ in range(2)]
        st["out"] = _pinned(lat)
        st["A"] = c2q.QplusQminus_eo()
    return st


# ---------------------------------------------------------------- one pass
def _download(field, buf):
    """A field into pinned host memory, in stream order."""
    c2q._check(field.system.lib.c2q_spinor_eo_download_async(field.h, buf.numpy(), None), field.system.h,
               field.system.lib)


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "cg":
        for x in st["x"]:
            x.zero()
        if case["nsrc"] == 1:
            c2q.cg(st["x"][0], st["A"], st["gf"], st["b"][0], st["params"], st["add"])
        else:
            c2q.cg_multi(st["x"], st["A"], st["gf"], st["b"], st["params"], st["add"])
        for x, o in zip(st["x"], st["out"]):
            _download(x, o)
        return st["out"]
    if kind == "bicgstab":
        st["x"][0].zero()
        c2q.bicgstab(st["x"][0], st["A"], st["gf"], st["b"][0], st["params"], st["add"])
        _download(st["x"][0], st["out"][0])
        return st["out"]
    if kind == "inversion":
        return c2q.perform_inversion(st["system"], st["gf"], st["source"], st["params"], st["add"])[0]
    if kind == "force":
        st["gm"].zero()
        c2q.calc_fermion_force(st["gm"], st["gf"], st["phi"], st["params"], st["add"])
        return st["gm"].download()
    if kind == "power":
        st["system"].set_link_format(case["rec12"])
        x, v = st["x"]
        c2q.copyData(x, st["start"])
        norms = []
        for _ in range(case["count"]):
            st["A"](v, st["gf"], x, st["add"])
            norms.append(math.sqrt(c2q.squarenorm(v)))
            c2q.sax(x, 1.0 / norms[-1], v)
        if case["precision"] == 64:
            _download(x, st["out"][0])
        else:
            st["full"].convert_from(x)
            _download(st["full"], st["out"][0])
        return {"norms": np.array(norms), "vector": st["out"][0]}
    tickets = []
    for (which, kappa, mu, nsrc, seed), out in zip(st["requests"], st["out"]):
        gid, la = st["gauges"][which]
        tickets.append(st["server"].submit(la, gid, kappa, mu, nsrc, seed, solutions=out))
    for t in tickets:
        r = st["server"].wait(t)
        if r["status"] != 0:
            raise RuntimeError("request failed with status %d" % r["status"])
    return st["out"]


# ---------------------------------------------------------------- work
def work(case):
    """Links and source read once, solution written once; the sweeps of a typical solve at 1392
    operations per output site."""
    kind, seo = case["kind"], case["ns"] ** 3 * case["nt"] // 2
    links, field = 8 * seo * 144, seo * 192
    n = case.get("nsrc", 1)
    if kind == "cg":
        return {"bytes": links + 2 * n * field, "flops": n * 90 * 4 * seo * 1392}
    if kind == "bicgstab":
        return {"bytes": links + 2 * field, "flops": 20 * 4 * seo * 1392}
    if kind == "inversion":
        return {"bytes": links + 4 * field, "flops": 20 * 4 * seo * 1392}
    if kind == "force":
        return {"bytes": links + field + 8 * seo * 64, "flops": 94 * 4 * seo * 1392}
    if kind == "power":
        size = case["precision"] / 64
        return {"bytes": size * (links * (2 / 3 if case["rec12"] else 1) + 2 * field),
                "flops": case["count"] * 4 * seo * 1392}
    b = f = 0
    lats = _two_lattices(case)
    for la in lats:
        b += 8 * la.seo * 144
    for which, _, _, nsrc, _ in _requests(case, 0):
        b += nsrc * lats[which].seo * 192
        f += nsrc * 90 * 4 * lats[which].seo * 1392
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------- the same in 64 bits with torch
class _Exact:
    """The even-odd twisted-mass operator on complex128 fields of shape (4, 3, Seo)."""

    # (1 - gamma_mu) keeps psi_a + c psi_p: the partner p and unit c of the upper spins a = 0, 1
    PROJ = [((2, 1), (3, 1)), ((3, 1j), (2, 1j)), ((3, 1), (2, -1)), ((2, 1j), (3, -1j))]

    def __init__(self, ns, nt, links, kappa, mu):
        self.kappa, self.mubar = kappa, 2 * kappa * mu
        site = torch.arange(ns ** 3 * nt, device="cuda")
        c = [site // ns ** 3, site % ns, site // ns % ns, site // ns ** 2 % ns]  # t, x, y, z
        ext = [nt, ns, ns, ns]
        par = (c[0] + c[1] + c[2] + c[3]) % 2
        self.sites = [site[par == p] for p in (0, 1)]
        self.U, self.to = [], []
        lk = links.reshape(-1, 4, 9)
        for p in (0, 1):
            s = self.sites[p]
            self.U.append([lk[s, m].t().contiguous() for m in range(4)])
            rows = []
            for m in range(4):
                for d in (1, -1):
                    n = [v[s] for v in c]
                    n[m] = (n[m] + d) % ext[m]
                    rows.append((n[1] + ns * (n[2] + ns * (n[3] + ns * n[0]))) // 2)
            self.to.append(rows)
        self.phase = [complex(math.cos(math.pi / nt), math.sin(math.pi / nt)), 1, 1, 1]

    def D(self, p, psi):
        """dslash_eo: the sites of parity p from a field on the other parity."""
        out = torch.zeros_like(psi)
        for m in range(4):
            for back in (0, 1):
                nb = self.to[p][2 * m + back]
                f = psi[:, :, nb]
                u = self.U[1 - p][m][:, nb] if back else self.U[p][m]
                w = complex(self.phase[m]).conjugate() if back else complex(self.phase[m])
                for a, (q, unit) in enumerate(self.PROJ[m]):
                    unit = -unit if back else unit
                    h = f[a] + unit * f[q]
                    for r in range(3):
                        if back:
                            s = u[r].conj() * h[0] + u[3 + r].conj() * h[1] + u[6 + r].conj() * h[2]
                        else:
                            s = u[3 * r] * h[0] + u[3 * r + 1] * h[1] + u[3 * r + 2] * h[2]
                        s = s * w
                        out[a, r] += s
                        out[q, r] += complex(unit).conjugate() * s
        return -self.kappa * out

    def R(self, psi, sign=1, inverse=False):
        f = torch.tensor([1, 1, -1, -1], dtype=torch.float64, device="cuda").reshape(4, 1, 1) * (1j * self.mubar * sign)
        return (1 - f) * psi / (1 + self.mubar ** 2) if inverse else (1 + f) * psi

    @staticmethod
    def g5(psi):
        return torch.cat([psi[:2], -psi[2:]])

    def A(self, psi, sign=1):
        return self.R(psi, sign) - self.D(1, self.R(self.D(0, psi), sign, True))

    def Q(self, psi, sign=1):
        return self.g5(self.A(psi, sign))

    def QQ(self, psi):
        return self.Q(self.Q(psi, -1), 1)

    def solve(self, b):
        """(Q+Q-)^-1 b by conjugate gradients."""
        dot = lambda x, y: float(torch.sum(x.real * y.real + x.imag * y.imag))  # noqa: E731
        x, r = torch.zeros_like(b), b.clone()
        p, rr = r.clone(), dot(r, r)
        stop = rr * 1e-26
        for _ in range(5000):
            v = self.QQ(p)
            al = rr / dot(p, v)
            x += al * p
            r -= al * v
            new = dot(r, r)
            if new < stop:
                break
            p = r + (new / rr) * p
            rr = new
        return x

    def solve_A(self, b):
        """A^-1 b = Q- (Q+Q-)^-1 g5 b, as Q- is the adjoint of Q+ = g5 A."""
        return self.Q(self.solve(self.g5(b)), -1)


def _cplx(t):
    return torch.view_as_complex(t.reshape(-1, 12, 2).contiguous()).t().reshape(4, 3, -1).contiguous()


def _flat(psi):
    return torch.view_as_real(psi.reshape(12, -1).t().contiguous()).reshape(-1, 24)


def _splitmix_z2(n, seed):
    """The server's seeded Z2 sources: one 64-bit word of signs per site."""
    with np.errstate(over="ignore"):
        gold = np.uint64(0x9E3779B97F4A7C15)
        s = np.uint64(seed ^ 0x5350494E4F52) ^ (np.arange(n, dtype=np.uint64) * gold + np.uint64(0xD1B54A32D192ED03))
        z = s + gold + gold  # the second word of each site's stream
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z ^= z >> np.uint64(31)
    bits = (z[:, None] >> np.arange(24, dtype=np.uint64)) & np.uint64(1)
    return torch.from_numpy(np.where(bits, -1.0, 1.0) / math.sqrt(2.0)).cuda()


def _force(E, y, x, p, gm, phases):
    """Adds the force of y (on parity p) and x (on the other) to gm[parity][mu] (8, Seo)."""
    y = _Exact.g5(y)
    for m in range(4):
        for back in (0, 1):
            nb = E.to[p][2 * m + back]
            f = x[:, :, nb]
            v = 0
            for a, (q, unit) in enumerate(E.PROJ[m]):
                unit = -unit if back else unit
                psi, phi = f[a] + unit * f[q], y[a] + unit * y[q]
                left, right = (psi, phi) if back else (phi, psi)
                v = v + left[:, None] * right[None].conj()
            u = (E.U[1 - p][m][:, nb] if back else E.U[p][m]).reshape(3, 3, -1)
            w = 2 * E.kappa * phases[m] * torch.einsum("rkn,qkn->rqn", u, v.conj())
            i = w.imag
            ae = torch.stack([-i[1, 0] - i[0, 1], w.real[1, 0] - w.real[0, 1], i[1, 1] - i[0, 0], -i[2, 0] - i[0, 2],
                              w.real[2, 0] - w.real[0, 2], -i[2, 1] - i[1, 2], w.real[2, 1] - w.real[1, 2],
                              (2 * i[2, 2] - i[0, 0] - i[1, 1]) / math.sqrt(3)])
            if back:
                gm[1 - p][m][:, nb] += ae
            else:
                gm[p][m] += ae


def exact(case, seed):
    ns, nt, kind = case["ns"], case["nt"], case["kind"]
    seo = ns ** 3 * nt // 2
    if kind == "serving":
        got, ops = [], {}
        for which, kappa, mu, nsrc, s in _requests(case, seed):
            la = _two_lattices(case)[which]
            if which not in ops:
                ops[which] = _links(la.ns, la.nt, case["eps"], seed + 7 * which)
            E = _Exact(la.ns, la.nt, ops[which], kappa, mu)
            got.append(torch.stack([_flat(E.solve(_cplx(_splitmix_z2(la.seo, s + k)))) for k in range(nsrc)]).cpu())
        return got
    if kind == "cg" and seo * case["nsrc"] > 4500000:
        return None
    E = _Exact(ns, nt, _links(ns, nt, case["eps"], seed), case["kappa"], case["mu"])
    if kind == "cg":
        return [_flat(E.solve(_cplx(_source(case["source"], seo, seed, k)))).cpu() for k in range(case["nsrc"])]
    if kind == "bicgstab":
        return [_flat(E.solve_A(_cplx(_source(case["source"], seo, seed)))).cpu()]
    if kind == "inversion":  # the reference's sign: -M^-1 b
        b = _source("gaussian", 2 * seo, seed)
        be, bo = (_cplx(b[E.sites[p]]) for p in (0, 1))
        xo = E.solve_A(bo - E.D(1, E.R(be, 1, True)))
        xe = E.R(be - E.D(0, xo), 1, True)
        b[E.sites[0]], b[E.sites[1]] = -_flat(xe), -_flat(xo)
        return b.cpu()
    if kind == "force":
        x = E.solve(_cplx(_source("gaussian", seo, seed)))
        y = E.Q(x, -1)
        gm = [[torch.zeros((8, seo), dtype=torch.float64, device="cuda") for _ in range(4)] for _ in (0, 1)]
        _force(E, y, -E.R(E.D(0, x), -1, True), 1, gm, E.phase)
        _force(E, -E.R(E.D(0, y), 1, True), x, 0, gm, E.phase)
        out = torch.zeros((2 * seo, 4, 8), dtype=torch.float64, device="cuda")
        for p in (0, 1):
            for m in range(4):
                out[E.sites[p], m] = gm[p][m].t()
        return out.reshape(-1, 8).cpu()
    x, norms = _cplx(_source("gaussian", seo, seed)), []
    for _ in range(case["count"]):
        v = E.QQ(x)
        norms.append(float(torch.linalg.vector_norm(v)))
        x = v / norms[-1]
    return {"norms": np.array(norms), "vector": _flat(x).cpu()}
