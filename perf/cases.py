"""The work users have this framework do, as measurable cases.

Every case goes through the entry points a program calls: ``GPUSolver`` (the residual-
interaction plugin ``calc_hamiltonian`` and the batched ``solve``, in the FP64 form and the
mixed form), the serving loop ``Server`` with its engines, and the finite-range
two-body-current set-up ``gamma_pieces``.

Ground states: the recorded 40S and 162Gd solutions in their own N_sh = 6 basis or
re-diagonalised in a larger full basis (N_sh up to 16), and the synthetic Bogoliubov state
of the large-basis stress configuration (N_sh = 20, Omega-only blocks).  They do not depend
on the seed; the omega points and the densities do.

Points lie on the CIRCLE contour (centre 10 MeV, radius 25 MeV) away from the real axis:
next to the axis the iteration does not converge, or wanders for so long that rounding
decides the digits it stops at.

Outputs: the strengths and cross terms a user reads, with the final state vectors where the
basis is small, the iteration table and the iteration counts of the FP64 form.  What the
mixed form computes with FP32 field evaluations is taken in single precision, its accuracy;
its iteration counts depend on that rounding and are not among the outputs.  ``exact``
repeats fields and FP64 iterations in numpy.
"""
import functools
import math
import os

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HELS = {"S40": "S40.hel", "Gd162": "Gd162.hel"}
INTERACTION = {"interaction_name": "SKOP", "require_self_consistency": False, "require_gauge_invariance": True,
               "force_j2_terms": False, "vpair_t0": -346.352, "override_cs0": 128.279, "override_csr": 0.0,
               "override_cds": 0.0}
ALPHA = float(np.float32(0.7))
# how near the ends of the half circle the points come (radians; 0.1 is 2.5 MeV off the axis)
LOW = {"solve": 0.2, "steps": 0.04, "serve": 0.08}


def listed():
    return [
        # the in-process plugin (one residual-interaction field) of a light nucleus in the
        # recorded basis: the smallest call, launches and copies
        dict(name="field_fp64_nsh6", kind="field", nucleus="S40", nsh=6, op="GT", k=0, mixed=False),
        # the same field at the production basis size
        dict(name="field_fp64_nsh16", kind="field", nucleus="Gd162", nsh=16, op="GT", k=1, mixed=False),
        # and in the arithmetic of the mixed form's increment evaluations
        dict(name="field_mixed_nsh16", kind="field", nucleus="Gd162", nsh=16, op="RS2", k=2, mixed=True),
        # one pnfam_main.x run: one omega point, reference defaults
        dict(name="point_fp64_nsh6", kind="solve", nucleus="S40", nsh=6, op="GT", k=0, points=1, mixed=False,
             history=50, alpha=ALPHA, temperature=0.0),
        # the half-circle contour of the oracle configuration: N_sh = 8, Broyden 7 and 0.4
        dict(name="contour_fp64_nsh8", kind="solve", nucleus="S40", nsh=8, op="GT", k=0, points=40, mixed=False,
             history=7, alpha=0.4, temperature=0.0),
        # statistical FAM (finite temperature, P and Q quadrants), a first-forbidden operator
        # with its cross terms
        dict(name="thermal_fp64_nsh6", kind="solve", nucleus="S40", nsh=6, op="RS1", k=1, points=5, mixed=False,
             history=50, alpha=ALPHA, temperature=1.5),
        # first iterations of the drop-in form at the production basis size (a restart slice)
        dict(name="steps_fp64_nsh16", kind="steps", nucleus="Gd162", nsh=16, op="RS1", k=0, points=9, mixed=False,
             steps=4, history=50),
        # the large-basis stress configuration: a fixed number of iterations, mixed form
        dict(name="steps_mixed_nsh20", kind="steps", nucleus="synthetic", nsh=20, op="GT", k=1, points=64, mixed=True,
             steps=4, history=7),
        # a mid-size basis with fewer points than fill the batched kernels
        dict(name="steps_mixed_nsh12", kind="steps", nucleus="Gd162", nsh=12, op="GT", k=1, points=11, mixed=True,
             steps=12, history=50),
        # a whole contour of one operator served in the mixed form: more points than slots
        dict(name="serve_mixed_nsh16", kind="serve", nucleus="Gd162", nsh=16, ops="GT0", points=56, slots=40),
        # several operators of one nucleus on the device together, short requests
        dict(name="serve_mixed_nsh8", kind="serve", nucleus="S40", nsh=8, ops="GT0,GT1,RS1-0", points=24, slots=16),
        # set-up of a finite-range two-body current (computed when no .tbc file exists)
        dict(name="two_body_nsh6", kind="tbc", nucleus="S40", nsh=6, k=0, use_p=False),
    ]


def draw(rng):
    kind = rng.choice(["field"] * 4 + ["solve"] * 3 + ["steps"] * 4 + ["serve"] * 2 + ["tbc"])
    nucleus = rng.choice(["S40", "Gd162"])
    op, k = rng.choice([("GT", 0), ("GT", 1), ("RS1", 0), ("RS1", 1), ("RS2", 2), ("P", 0), ("R", 1)])
    if kind == "field":
        return dict(kind=kind, nucleus=nucleus, nsh=rng.randint(6, 16), op=op, k=k, mixed=rng.random() < 0.5)
    if kind == "solve":
        return dict(kind=kind, nucleus="S40", nsh=rng.choice([6, 7, 8]), op=op, k=k, points=_log_int(rng, 1, 24),
                    mixed=False, history=rng.choice([20, 50]), alpha=ALPHA, temperature=rng.choice([0.0, 0.0, 1.0]))
    if kind == "steps":
        mixed = rng.random() < 0.6
        nsh = rng.randint(7, 16)
        most = min(64, 200000 // nsh ** 4 + 8) if mixed else min(40, 60000 // nsh ** 4 + 8)
        return dict(kind=kind, nucleus=nucleus, nsh=nsh, op=op, k=k, points=_log_int(rng, 1, most), mixed=mixed,
                    steps=rng.randint(3, 6), history=50)
    if kind == "serve":
        return dict(kind=kind, nucleus="S40", nsh=rng.choice([6, 8, 10]), ops=rng.choice(["GT0", "GT0,GT1", "GT1,RS2-2"]),
                    points=_log_int(rng, 5, 40), slots=rng.choice([9, 16, 24]))
    return dict(kind=kind, nucleus=nucleus, nsh=rng.choice([4, 5, 6, 7]), k=rng.choice([0, 1]),
                use_p=rng.random() < 0.4)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# ---------------------------------------------------------------------------
# what a program has in hand: ground state, couplings, operator
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _ground_state(nucleus, nsh):
    from pynfam_gb300.synthetic import bogoliubov_nucleus, ground_state
    path = os.path.join(ROOT, "tests", "golden", HELS.get(nucleus, "Gd162.hel"))
    if nucleus == "synthetic":
        return bogoliubov_nucleus(path, nsh, seed=3, parity=False)
    return ground_state(path, nsh)


@functools.lru_cache(maxsize=None)
def _operator(nucleus, nsh, op, k):
    from pynfam_gb300.namelist import defaults
    from pynfam_gb300.pnfam_setup import setup_case
    nml = defaults()
    nml["interaction"].update(INTERACTION)
    nml["ext_field"].update(operator_name=op, operator_k=k, beta_type="-", compute_crossterms=True)
    return setup_case(nml, None, hfb=_ground_state(nucleus, nsh))


def _occupations(case, c):
    from pynfam_gb300.statistics import thermal_occupations
    t = case.get("temperature", 0.0)
    return thermal_occupations(c.hfb, t) if t else None


def _points(n, seed, low):
    """n points of the CIRCLE contour's upper half, shifted along it by the seed."""
    rng = np.random.default_rng([seed, 17])
    t = low + (math.pi - 2 * low) * (np.arange(n) + rng.uniform(0.05, 0.95, n)) / n
    return 10.0 + 25.0 * np.exp(1j * t)


def _densities(c, seed):
    """Perturbed densities of the size that the iteration meets, in the plugin's layout."""
    rng = np.random.default_rng([seed, 29])
    n = c.F.mat.nelem
    return [0.05 * (rng.standard_normal(n) + 1j * rng.standard_normal(n)) for _ in range(4)]


def _ops(case):
    out = []
    for s in case["ops"].split(","):
        out.append((s[:-1].rstrip("-"), int(s[-1])))
    return out


def prepare(case, seed):
    from pynfam_gb300.solver import GPUSolver
    if case["kind"] == "tbc":
        import dataclasses
        c = _operator(case["nucleus"], case["nsh"], "GT", case["k"])
        # the ground state's density matrices are the input: another seed, another pairing tail
        h = dataclasses.replace(c.hfb, Vn=_scaled(c.hfb.Vn, seed), Vp=_scaled(c.hfb.Vp, seed + 1))
        return dict(case=case, hfb=h, F=c.F)
    if case["kind"] == "serve":
        cs = {o: _operator(case["nucleus"], case["nsh"], *o) for o in _ops(case)}
        solvers = {}
        for o, c in cs.items():
            solvers[o] = GPUSolver(c.hfb, c.couplings)
            solvers[o].set_operator(c.F, c.G)
        return dict(case=case, solvers=solvers, quench={o: c.quench for o, c in cs.items()},
                    omegas={o: _points(case["points"], seed + 31 * i, LOW["serve"]) for i, o in enumerate(cs)})
    c = _operator(case["nucleus"], case["nsh"], case["op"], case["k"])
    g = GPUSolver(c.hfb, c.couplings, occupations=_occupations(case, c))
    g.set_operator(c.F, c.G)
    state = dict(case=case, solver=g, quench=c.quench)
    if case["kind"] == "field":
        state["rho"] = _densities(c, seed)
    else:
        state["omegas"] = _points(case["points"], seed, LOW[case["kind"]])
    return state


def _scaled(V, seed):
    f = 1.0 - 0.02 * np.random.default_rng([seed, 41]).random()
    return [f * v for v in V]


def run(state):
    case = state["case"]
    return {"field": _run_field, "solve": _run_solve, "steps": _run_steps, "serve": _run_serve,
            "tbc": _run_tbc}[case["kind"]](case, state)


def _run_field(case, s):
    out = s["solver"].calc_hamiltonian(*s["rho"], mixed=case["mixed"])
    return [x.astype(np.complex64) for x in out] if case["mixed"] else list(out)


def _run_solve(case, s):
    r = s["solver"].solve(s["omegas"], max_iter=200, eps=1e-7, broyden_m=case["history"], quench=s["quench"],
                          alpha_mix=case["alpha"], return_state=True)
    return dict(S=r.re_S + 1j * r.im_S, iters=r.iters, state=r.state)


def _run_steps(case, s):
    small = case["nsh"] <= 12
    r = s["solver"].solve(s["omegas"], max_iter=case["steps"], eps=1e-13, broyden_m=case["history"],
                          quench=s["quench"], history=not case["mixed"], precision=1 if case["mixed"] else 0,
                          return_state=small)
    S = r.re_S + 1j * r.im_S
    if case["mixed"]:
        out = dict(S=S.astype(np.complex64))
    else:
        out = dict(S=S, table=r.hist)
    if small:
        out["state"] = r.state.astype(np.float32) if case["mixed"] else r.state
    return out


def _run_serve(case, s):
    from pynfam_gb300.serve import Request, Server

    def engine(key, slots):
        return s["solvers"][key].engine(slots, max_iter=200, eps=1e-8, broyden_m=50, quench=s["quench"][key],
                                        precision=1, settle=8, near_exp=4, switch_exp=5)
    keys = list(s["solvers"])
    server = Server(engine, lambda key, n: 1, slots=case["slots"], budget_bytes=len(keys))
    out, _ = server.run([Request(i, k, s["omegas"][k], 0.0) for i, k in enumerate(keys)])
    S = {i: np.zeros((case["points"], s["solvers"][k].nops), dtype=np.complex64) for i, k in enumerate(keys)}
    for o in out:
        S[o.rid][o.index] = o.S
    return [S[i] for i in range(len(keys))]


def _run_tbc(case, s):
    from pynfam_gb300.finite_range import gamma_pieces
    return gamma_pieces(s["hfb"], s["F"], use_p=case["use_p"])


# ---------------------------------------------------------------------------
# what one pass cannot do without
# ---------------------------------------------------------------------------
def _sizes(nucleus, nsh, op, k):
    c = _operator(nucleus, nsh, op, k)
    h, fc = c.hfb, c.F.mat.cols
    pairs = [(int(h.db[i]), int(h.db[j])) for i, j in enumerate(fc) if j >= 0]
    n = dict(nxy=sum(a * b for a, b in pairs), S3=sum(a * a * b for a, b in pairs), nghl=int(h.nghl),
             dqp=int(h.dqp), ground=4 * int((np.asarray(h.db) ** 2).sum()), nops=1 + len(c.G))
    # the products of one field on the mesh (a sum over the states of one side per mesh point
    # would be 88 nghl nxy): the mesh and the oscillator functions are products of a z and a
    # radial part, so one side's sums cost the nodes of one direction per matrix element
    node = int(round(math.sqrt(n["nghl"])))
    n["field"] = 2 * (2 * 2 * 2 * 2 * node) * n["nxy"] * 2 + 2600 * n["nghl"]
    # QP <-> SP transforms, Re and Im: four first products shared, eight second ones, twice
    n["transform"] = 96 * n["S3"]
    return n


def work(case):
    kind = case["kind"]
    if kind == "tbc":
        z = _sizes(case["nucleus"], case["nsh"], "GT", case["k"])
        terms = math.comb(case["nsh"] + 3, 3)
        return dict(bytes=8.0 * (6 * z["nxy"] + z["ground"] / 2), flops=2.0 * 84 * z["nxy"] * terms)
    if kind == "serve":
        total = dict(bytes=0.0, flops=0.0)
        for o in _ops(case):
            z = _sizes(case["nucleus"], case["nsh"], *o)
            its = 30   # evaluations of a typical point of the contour
            total["bytes"] += 8.0 * (z["ground"] + 5 * z["dqp"] * z["nghl"]) + 16.0 * case["points"] * (1 + z["nops"])
            total["flops"] += case["points"] * its * (z["transform"] + z["field"] + 4 * 4 * z["nxy"] * its)
        return total
    z = _sizes(case["nucleus"], case["nsh"], case["op"], case["k"])
    basis = 8.0 * 5 * z["dqp"] * z["nghl"]
    if kind == "field":
        return dict(bytes=basis + 16.0 * 8 * z["nxy"], flops=z["field"])
    its = case["steps"] - 1 if kind == "steps" else 25
    nq = 4 if case.get("temperature") else 2
    per = z["transform"] * nq / 2 + z["field"] + 4 * 2 * nq * z["nxy"] * its
    state = 8.0 * 2 * nq * z["nxy"] if case["nsh"] <= 12 else 0.0
    return dict(bytes=basis + 8.0 * z["ground"] + case["points"] * (state + 16.0 * (1 + z["nops"])),
                flops=case["points"] * its * per)


# ---------------------------------------------------------------------------
# the same numbers in plain numpy, 64 bits
# ---------------------------------------------------------------------------
EPS = np.zeros((4, 4, 4))
for _p, _s in (((1, 2, 3), 1), ((2, 3, 1), 1), ((3, 1, 2), 1), ((1, 3, 2), -1), ((3, 2, 1), -1), ((2, 1, 3), -1)):
    EPS[_p] = _s


def _sigma(sa, sb):
    """(1, sigma_r, sigma_phi, sigma_z) between spins sa and sb."""
    return np.array([1.0, 0.0, 0.0, sa] if sa == sb else [0.0, 1.0, 1j * sa, 0.0], dtype=complex)


class _Mesh:
    def __init__(self, c):
        h = self.h = c.hfb
        self.cp = c.couplings
        self.v = np.stack([h.wf, h.wfdr, 1j * h.wfdp, h.wfdz])   # phi and its gradient
        self.st = np.asarray(h.isstart)

    def segments(self, cols):
        """(rows, columns, spins) of the spin-pure parts of every block."""
        h = self.h
        for i, j in enumerate(cols):
            if j < 0:
                continue
            a, b, nu, nv = self.st[i], self.st[j], h.num_spin_up[i], h.num_spin_up[j]
            for ra, sa in ((slice(a, a + nu), 1), (slice(a + nu, a + h.db[i]), -1)):
                for rb, sb in ((slice(b, b + nv), 1), (slice(b + nv, b + h.db[j]), -1)):
                    if ra.stop > ra.start and rb.stop > rb.start:
                        yield ra, rb, sa, sb

    def field(self, rho, rcols, kap, kcols, dcols):
        """(h in rho's structure, Delta in dcols) of dense rho and kappa: the derivative of
        the Skyrme functional's time-even and time-odd parts, written with
        K[m, n, nu] = sum_ab v_a[m] rho_ab conj(v_b[n]) sigma_nu(s_a, s_b), m = 0: phi,
        1..3: its gradient."""
        h, cp, v, w = self.h, self.cp, self.v, self.v.conj()
        n = h.nghl
        K = np.zeros((4, 4, 4, n), dtype=complex)
        for ra, rb, sa, sb in self.segments(rcols):
            sg = _sigma(sa, sb)
            on = np.nonzero(sg)[0]
            for m in range(4):
                x = v[m, ra].T @ rho[ra, rb]
                for q in range(4):
                    t = np.einsum("rb,br->r", x, w[q, rb])
                    for nu in on:
                        K[m, q, nu] += sg[nu] * t
        K *= h.wdcori
        G = range(1, 4)
        r, s = K[0, 0, 0], K[0, 0]
        kin = K[1, 1] + K[2, 2] + K[3, 3]
        j = [0] + [0.5j * (K[0, m, 0] - K[m, 0, 0]) for m in G]
        J = np.zeros((4, 4, n), dtype=complex)
        for m in G:
            for u in G:
                J[m, u] = 0.5j * (K[0, m, u] - K[m, 0, u])
        F = [0] + [0.5 * sum(K[m, u, u] + K[u, m, u] for u in G) for m in G]
        div = sum(K[u, 0, u] + K[0, u, u] for u in G)
        JV = np.einsum("lmn,mnr->lr", EPS, J)
        tr = J[1, 1] + J[2, 2] + J[3, 3]
        lap = [2 * (cp.cdrho if u == 0 else cp.cds) * s[u] for u in range(4)]
        M = np.zeros_like(K)
        M[0, 0, 0] = 2 * cp.crho * r + cp.ctau * kin[0]
        for u in G:
            M[0, 0, u] = 2 * cp.cs * s[u] + cp.ct * kin[u] + cp.cf * F[u]
        for m in G:
            M[m, m, 0] += cp.ctau * r + 2 * lap[0]
            M[0, m, 0] += 1j * cp.cj * j[m] - cp.crdj * JV[m]
            M[m, 0, 0] += -1j * cp.cj * j[m] - cp.crdj * JV[m]
            for u in G:
                M[m, m, u] += cp.ct * s[u] + 2 * lap[u]
                M[m, u, u] += 0.5 * cp.cf * s[m]
                M[u, m, u] += 0.5 * cp.cf * s[m]
                dJ = 2 * cp.ctj0 * tr * (m == u) + 2 * cp.ctj1 * np.einsum("l,lr->r", EPS[:, m, u], JV)
                dJ = dJ + 2 * cp.ctj2 * (0.5 * (J[m, u] + J[u, m]) - tr / 3.0 * (m == u))
                M[0, m, u] += 0.5j * dJ
                M[m, 0, u] -= 0.5j * dJ
            M[m, 0, m] += 2 * cp.cgs * div
            M[0, m, m] += 2 * cp.cgs * div
            for a in G:
                for b in G:
                    e = EPS[m, a, b]
                    if e:
                        M[m, a, b] += 1j * e * cp.crdj * r
                        M[a, b, 0] += 1j * e * cp.csdj * s[m]
                        M[a, 0, b] += e * cp.csdj * j[m]
                        M[0, a, b] += e * cp.csdj * j[m]
        out = np.zeros_like(rho)
        for ra, rb, sa, sb in self.segments(rcols):
            sg = _sigma(sb, sa)
            Ms = np.einsum("u,mqur->mqr", sg, M)
            Ls = sum(sg[u] * lap[u] for u in range(4))
            for q in range(4):
                x = sum(Ms[m, q] * v[m, rb] for m in range(4))
                if q == 0:
                    x = x + Ls * h.wfd2_all[rb]
                out[ra, rb] += 2 * w[q, ra] @ x.T
            out[ra, rb] += 2 * h.wfd2_all[ra] @ (Ls * h.wf[rb]).T
        # pairing
        k = {}
        for ra, rb, sa, sb in self.segments(kcols):
            t = 2 * np.einsum("ar,ab,br->r", h.wf[ra], kap[ra, rb], h.wf[rb], optimize=True) * h.wdcori
            k[sa, sb] = k.get((sa, sb), 0) + t
        o = np.zeros(n, dtype=complex)
        pp, pm, mp, mm = (k.get(x, o) for x in ((1, 1), (1, -1), (-1, 1), (-1, -1)))
        rb_, sz = pm - mp, pm + mp
        sr, sp = mm - pp, -1j * (mm + pp)
        D = {(1, 1): cp.cspair * (sr - 1j * sp), (-1, 1): -cp.cpair * rb_ - cp.cspair * sz,
             (1, -1): cp.cpair * rb_ - cp.cspair * sz, (-1, -1): cp.cspair * (-sr - 1j * sp)}
        del_ = np.zeros_like(rho)
        for ra, rb, sa, sb in self.segments(dcols):
            del_[ra, rb] = 2 * h.wf[ra] @ (D[sa, sb] * h.wf[rb]).T
        return out, del_


def _structures(c):
    """Block columns of F, X, Y, X^T, Y^T."""
    h = c.hfb
    fc = np.asarray(c.F.mat.cols)
    tr = np.array([h.partner(i) for i in range(h.nb)])
    x = np.where(fc >= 0, tr[fc], -1)
    y = fc[tr]

    def inverse(cols):
        inv = np.full(len(cols), -1)
        for i, j in enumerate(cols):
            if j >= 0:
                inv[j] = i
        return inv
    return fc, x, y, inverse(x), inverse(y)


def _dense(c, cols, flat):
    h = c.hfb
    out = np.zeros((h.dqp, h.dqp), dtype=np.asarray(flat).dtype)
    st, p = np.asarray(h.isstart), 0
    for i, j in enumerate(cols):
        if j >= 0:
            d, e = int(h.db[i]), int(h.db[j])
            out[st[i]:st[i] + d, st[j]:st[j] + e] = flat[p:p + d * e].reshape(d, e, order="F")
            p += d * e
    return out


def _flat(c, cols, m):
    h, st = c.hfb, np.asarray(c.hfb.isstart)
    return np.concatenate([m[st[i]:st[i] + h.db[i], st[j]:st[j] + h.db[j]].reshape(-1, order="F")
                           for i, j in enumerate(cols) if j >= 0])


def _exact_field(case, seed):
    c = _operator(case["nucleus"], case["nsh"], case["op"], case["k"])
    fc, xc, yc, xt, yt = _structures(c)
    mesh = _Mesh(c)
    rp, kp, rn, km = _densities(c, seed)
    hp, dp = mesh.field(_dense(c, fc, rp), fc, _dense(c, xt, kp), xt, xc)
    hn, dm = mesh.field(_dense(c, fc, rn), fc, _dense(c, yt, km), yt, yc)
    return [_flat(c, fc, hp), _flat(c, xc, dp), _flat(c, fc, hn), _flat(c, yc, dm)]


class _Iteration:
    """dR -> G o (q H(dR) + F) on dense matrices (beta-)."""

    def __init__(self, case):
        c = self.c = _operator(case["nucleus"], case["nsh"], case["op"], case["k"])
        h = c.hfb
        self.fc, self.xc, self.yc, self.xt, self.yt = _structures(c)
        tr = [h.partner(i) for i in range(h.nb)]
        flat = lambda B: np.concatenate([b.reshape(-1, order="F") for b in B])
        eye = list(range(h.nb))
        self.U = {s: _dense(c, eye, flat(B)) for s, B in (("L", h.Up), ("R", h.Un))}
        self.V = {s: _dense(c, tr, flat(B)) for s, B in (("L", h.Vp), ("R", h.Vn))}
        self.occ = _occupations(case, c)
        self.mesh = _Mesh(c)
        qc = np.array([tr[j] if j >= 0 else -1 for j in self.yc])
        self.cols = [self.xc, self.yc] + ([self.fc, qc] if self.occ else [])
        z = np.zeros((h.dqp, h.dqp))
        self.ops = [self._qp(_dense(c, self.fc, g.mat.flatten()) + 0j, z, z, z) for g in [c.F] + list(c.G)]

    def _qp(self, h11, h12, m21, m22):
        UL, VL, UR, VR = self.U["L"].T, self.V["L"].T, self.U["R"], self.V["R"]
        m21, m22 = m21.conj(), m22.T
        out = [UL @ (h11 @ VR + h12 @ UR) - VL @ (m21 @ VR + m22 @ UR),
               -VL @ (h11 @ UR + h12 @ VR) + UL @ (m21 @ UR + m22 @ VR)]
        if self.occ:
            out += [UL @ (h11 @ UR + h12 @ VR) - VL @ (m21 @ UR + m22 @ VR),
                    -VL @ (h11 @ VR + h12 @ UR) + UL @ (m21 @ VR + m22 @ UR)]
        return out

    def field(self, q):
        UL, VL, URt, VRt = self.U["L"], self.V["L"], self.U["R"].T, self.V["R"].T
        X, Y = q[0], q[1]
        P, Q = (q[2], q[3]) if self.occ else (0 * X, 0 * Y)
        ux, vy, up, vq = UL @ X, VL @ Y, UL @ P, VL @ Q
        vx, uy, vp, uq = VL @ X, UL @ Y, VL @ P, UL @ Q
        rho = ux @ VRt - vy @ URt + up @ URt - vq @ VRt
        kp = (-ux @ URt + vy @ VRt - up @ VRt + vq @ URt).T
        km = (vx @ VRt - uy @ URt + vp @ URt - uq @ VRt).T.conj()
        rn = (-vx @ URt + uy @ VRt - vp @ VRt + uq @ URt).T
        h11, h12 = self.mesh.field(rho, self.fc, kp, self.xt, self.xc)
        m22, m21 = self.mesh.field(rn, self.fc, km, self.yt, self.yc)
        return self._qp(h11, h12, m21, m22)

    def green(self, w):
        h = self.c.hfb
        e1, e2 = h.Ep[:, None], h.En[None, :]
        with np.errstate(divide="ignore", invalid="ignore"):
            G = [-1 / (e1 + e2 - w), -1 / (e1 + e2 + w)]
            if self.occ:
                f1, f2 = self.occ[0][:, None], self.occ[1][None, :]
                G = [(1 - f1 - f2) * G[0], (1 - f1 - f2) * G[1], (f2 - f1) * (-1 / (e1 - e2 - w)),
                     (f2 - f1) * (-1 / (e1 - e2 + w))]
        return [_flat(self.c, cols, g) for cols, g in zip(self.cols, G)]

    def pack(self, flats):
        """The restart order: Re X, Re Y, Im X, Im Y[, Re P, Re Q, Im P, Im Q]."""
        return np.concatenate([np.concatenate([a.real, b.real, a.imag, b.imag])
                               for a, b in zip(flats[::2], flats[1::2])])

    def unpack(self, x):
        parts, out = x.reshape(-1, self.c.F.mat.nelem), []
        for g in range(0, len(parts), 4):
            out += [parts[g] + 1j * parts[g + 2], parts[g + 1] + 1j * parts[g + 3]]
        return out

    def solve(self, w, max_iter, eps, M, alpha):
        c, G = self.c, self.green(w)
        F = [[_flat(c, cols, f) for cols, f in zip(self.cols, op)] for op in self.ops]
        x = np.zeros(2 * len(self.cols) * c.F.mat.nelem)
        df, dv, table, its = {}, {}, [(1.0, 0.0, 0.0)], -1
        S = np.zeros(len(F), dtype=complex)
        for it in range(max_iter):
            if it:
                H = self.field([_dense(c, cols, q) for cols, q in zip(self.cols, self.unpack(x))])
                H = [c.quench * _flat(c, cols, m) for cols, m in zip(self.cols, H)]
            else:
                H = [0.0] * len(self.cols)
            f = self.pack([g * (a + b) for g, a, b in zip(G, H, F[0])]) - x
            si = np.max(np.abs(f))
            step = alpha * f
            if it >= 1:
                # the columns in use: those of the last M steps, in their slots
                if it >= 2:
                    p = (it - 2) % M
                    df[p], dv[p] = f - df[p], x - dv[p]
                    nrm = np.linalg.norm(df[p])
                    df[p], dv[p] = df[p] / nrm, dv[p] / nrm
                use = list(range(min(it - 1, M)))
                if use:
                    A = np.stack([df[k] for k in use])
                    B = A @ A.T
                    B[np.diag_indices_from(B)] = 1.0 + 1e-4
                    g = np.linalg.solve(B, A @ f)
                    for k in use:
                        step = step - g[k] * (dv[k] + alpha * df[k])
                p = (it - 1) % M
                df[p], dv[p] = f.copy(), x.copy()
            x = x + step
            q = self.unpack(x)
            S = np.array([-sum(np.dot(a.real, b) for a, b in zip(op, q)) / math.pi for op in F])
            table.append((si, S[0].real, S[0].imag))
            if si < eps:
                its = it + 1
                break
        return S, its, x, np.array(table)


def exact(case, seed):
    if case["kind"] == "field":
        return _exact_field(case, seed)
    cost = case.get("points", 0) * case["nsh"] ** 3 * case.get("steps", 25)
    if case["kind"] == "serve":
        cost *= len(_ops(case))
    if case["kind"] == "tbc" or case["nsh"] > 8 or cost > 30000:
        return None   # over about 20 seconds
    if case["kind"] == "serve":
        # the fixed points (the last steps are below 1e-10)
        out = []
        for i, (op, k) in enumerate(_ops(case)):
            it = _Iteration(dict(case, op=op, k=k))
            out.append(np.array([it.solve(w, 200, 1e-10, 50, ALPHA)[0]
                                 for w in _points(case["points"], seed + 31 * i, LOW["serve"])]))
        return out
    it = _Iteration(case)
    if case["kind"] == "solve":
        r = [it.solve(w, 200, 1e-7, case["history"], case["alpha"]) for w in _points(case["points"], seed, LOW["solve"])]
        return dict(S=np.array([x[0] for x in r]), iters=None, state=np.array([x[2] for x in r]))
    r = [it.solve(w, case["steps"], 1e-13, case["history"], ALPHA) for w in _points(case["points"], seed, LOW["steps"])]
    out = dict(S=np.array([x[0] for x in r]), state=np.array([x[2] for x in r]))
    if not case["mixed"]:
        out["table"] = np.array([x[3] for x in r])
    return out
