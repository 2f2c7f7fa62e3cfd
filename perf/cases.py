"""The work that users of this package have it do, as timed cases.

Each case is one pass through a public entry point on inputs that such a
program has on the GPU already: the drop-in operators of ``_C`` and ``ops``,
the fermion force, the fermion action and its gradient on a batched PCG solver
whose plan the caller keeps, several lattices' solves in one launch, the
estimator's noise solves and bond-bond correlators, and whole HMC proposals.
Mixed-precision solves are followed, as in the sampler and the estimator, by
what takes their solutions in single precision.
Fields are those of the simulations: the pi-flux saddle point with static and
slice-to-slice fluctuations; pseudofermions and noise vectors are drawn as the
sampler and the estimator draw them.  Lattices follow the package's habit of
Ltau near 10 L at dtau = 0.1.  Solvers take the library's own launch shapes,
so that a case does not depend on what an earlier process tuned.
"""
from __future__ import annotations

import math

import torch

from qed_fermion_b200 import _C, ops, precon
from qed_fermion_b200.estimator import StochaticEstimator
from qed_fermion_b200.force import fermion_action
from qed_fermion_b200.hmc import HmcSampler, kernel_to_ref
from qed_fermion_b200.observables import BondBond
from qed_fermion_b200.solver import PcgSolver, System

DTAU = 0.1
RTOL = 1e-10
COMPLEX = {"c64": torch.complex64, "c128": torch.complex128}
REAL = {"c64": torch.float32, "c128": torch.float64}
# lattice sides that the slice kernels take: even ones up to 48, then those
# whose rows divide into taller tiles; 16, 32 and 64, whose rows fill a warp
# and have an operator of their own, are not drawn
SIDES = [s for s in range(6, 50, 2) if s not in (16, 32)] + [52, 54, 56, 60, 66]


def listed():
    return [
        # the smallest call of the reference's own CG loop on the drop-in operator: latency
        {"name": "mhm_small", "kind": "mhm", "L": 10, "Nt": 100, "nvec": 2, "dtype": "c64"},
        # M^dag M of eight chains on the production lattice
        {"name": "mhm_large", "kind": "mhm", "L": 48, "Nt": 480, "nvec": 8, "dtype": "c64"},
        # the same operator of the plain FP64 path
        {"name": "mhm_double", "kind": "mhm", "L": 36, "Nt": 360, "nvec": 4, "dtype": "c128"},
        # the preconditioner between the operator calls of the drop-in loop, ragged in tau
        {"name": "precon", "kind": "precon", "L": 36, "Nt": 359, "nvec": 8, "dtype": "c64"},
        # the fermion force of two chains after a solve
        {"name": "force", "kind": "force", "L": 48, "Nt": 480, "nvec": 2, "dtype": "c64"},
        # the fermion action and its gradient on the plain FP64 path, a mid-size lattice
        {"name": "solve_double", "kind": "solve", "L": 24, "Nt": 240, "nrhs": 2, "mode": "fp64"},
        # the solve that HMC spends its time on, then its force: two chains, mixed precision
        {"name": "solve_hmc", "kind": "solve", "L": 48, "Nt": 480, "nrhs": 2, "mode": "mixed"},
        # one chain on the largest lattice, forward and backward
        {"name": "solve_largest", "kind": "solve", "L": 66, "Nt": 660, "nrhs": 1, "mode": "mixed"},
        # sixteen independent lattices of uneven size solved in one launch, then each one's force
        {"name": "solve_uneven", "kind": "batch", "Ls": "12,18,24,30", "each": 4, "mode": "mixed"},
        # the estimator's noise solves: 64 Z2 vectors on one field
        {"name": "estimator", "kind": "noise", "L": 36, "Nt": 360, "nrhs": 64, "mode": "mixed"},
        # its bond-bond correlators over all pairs of 20 vectors
        {"name": "correlators", "kind": "bond", "L": 30, "Nt": 300, "nrhs": 20, "dtype": "c128"},
        # a whole HMC proposal of two chains on a small lattice: launches and short solves
        {"name": "proposal", "kind": "proposal", "L": 10, "Nt": 100, "chains": 2, "steps": 5},
    ]


def _log_pick(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi):
    return min((s for s in SIDES if lo <= s <= hi), key=lambda s, x=_log_pick(rng, lo, hi): abs(s - x))


def draw(rng):
    kind = rng.choice(["mhm", "mhm", "precon", "force", "force", "solve", "solve", "solve", "batch", "noise", "bond",
                       "proposal"])
    if kind in ("mhm", "precon", "force"):
        L = _side(rng, 6, 66)
        Nt = rng.randint(6 * L, 11 * L)
        most = max(1, min(16, 9_000_000 // (L * L * Nt)))
        return {"kind": kind, "L": L, "Nt": Nt, "nvec": rng.randint(1, most), "dtype": rng.choice(["c64", "c128"])}
    if kind == "solve":
        L = _side(rng, 8, 66)
        Nt = rng.randint(7 * L, 10 * L)
        most = max(1, min(6, 3_000_000 // (L * L * Nt)))
        return {"kind": kind, "L": L, "Nt": Nt, "nrhs": rng.randint(1, most),
                "mode": rng.choice(["mixed", "mixed", "fp64"]) if L <= 48 else "mixed"}
    if kind == "batch":
        Ls = sorted(rng.sample([8, 10, 12, 14, 18, 20, 24, 28, 30], rng.randint(2, 4)))
        return {"kind": kind, "Ls": ",".join(map(str, Ls)), "each": rng.randint(1, 4), "mode": "mixed"}
    if kind == "noise":
        L = _side(rng, 10, 36)
        return {"kind": kind, "L": L, "Nt": rng.randint(8 * L, 10 * L), "nrhs": rng.randint(4, 48), "mode": "mixed"}
    if kind == "bond":
        L = _side(rng, 8, 30)
        return {"kind": kind, "L": L, "Nt": rng.randint(8 * L, 10 * L), "nrhs": rng.randint(4, 20),
                "dtype": rng.choice(["c64", "c128"])}
    L = _side(rng, 6, 20)
    return {"kind": kind, "L": L, "Nt": rng.randint(max(26, 7 * L), 10 * L), "chains": rng.randint(1, 3),
            "steps": rng.randint(2, 5)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed, k=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + k)


def _field(L, Nt, n, g):
    """Angles [n, Nt, L, L, 2]: the pi-flux saddle point, a static deviation and slice-to-slice noise."""
    i = torch.arange(L, device="cuda")
    sign = (1 - 2 * ((i.view(-1, 1) + i.view(1, -1)) % 2)).double() * (math.pi / 4)
    stag = torch.stack([sign, -sign], dim=-1)
    static = 0.05 * torch.randn((n, 1, L, L, 2), device="cuda", dtype=torch.float64, generator=g)
    moving = 0.05 * torch.randn((n, Nt, L, L, 2), device="cuda", dtype=torch.float64, generator=g)
    # what a float32 simulation holds, also for the double-precision cases
    return (stag + static + moving).float()


def _gauss(rows, n, g):
    return torch.randn((rows, n), device="cuda", dtype=torch.complex128, generator=g) / math.sqrt(2)


def _systems(case):
    if case["kind"] == "batch":
        Ls = [int(s) for s in case["Ls"].split(",")]
        return [(L, 10 * L, 1, False) for L in Ls for _ in range(case["each"])]
    return [(case["L"], case["Nt"], case["nrhs"], case["kind"] == "noise")]


def _solve_inputs(case, seed):
    """Packed angles and right-hand sides M^dag R of every system."""
    phis, bs = [], []
    for k, (L, Nt, nrhs, shared) in enumerate(_systems(case)):
        g = _gen(seed, k)
        phi = _field(L, Nt, 1 if shared else nrhs, g)
        R = _gauss(nrhs, L * L * Nt, g)
        phis.append(phi.reshape(-1))
        bs.append(_Exact(phi, L, 1 if shared else nrhs).mh(R).reshape(-1))
    return torch.cat(phis), torch.cat(bs)


def _noise(case, seed):
    g = _gen(seed)
    phi = _field(case["L"], case["Nt"], 1, g)
    eta = torch.randint(0, 2, (case["nrhs"], case["L"] ** 2 * case["Nt"]), device="cuda", generator=g) * 2 - 1
    return phi, eta.to(torch.complex128)


def _propagated(eta, L, Nt, g):
    """Vectors like G eta: the noise, its neighbours in space and time, and a remainder."""
    e = eta.view(-1, Nt, L, L)
    out = 0.5 * e
    for dim, w in ((1, 0.3), (2, 0.12j), (3, 0.12)):
        out = out + w * torch.roll(e, 1, dim) - w * 0.5 * torch.roll(e, -1, dim)
    return (out + 0.1 * torch.randn(e.shape, device="cuda", dtype=torch.complex128, generator=g)).reshape(eta.shape)


def _proposal_inputs(case, seed):
    g = _gen(seed)
    L, Nt, n = case["L"], case["Nt"], case["chains"]
    boson = kernel_to_ref(_field(L, Nt, n, g).reshape(n, -1), L, Nt)
    p0 = torch.randn(boson.shape, device="cuda", generator=g)
    return boson, p0, _gauss(n, L * L * Nt, g)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("mhm", "precon", "force"):
        g = _gen(seed)
        L, Nt, n, dt = case["L"], case["Nt"], case["nvec"], case["dtype"]
        s["phi"] = _field(L, Nt, n, g).to(REAL[dt]).reshape(n, -1)
        s["x"] = _gauss(n, L * L * Nt, g).to(COMPLEX[dt])
        if kind == "precon":
            s["tau"] = precon.to_device(precon.builtin_tau_csr(Nt), s["x"].device)
    elif kind in ("solve", "batch"):
        phi, b = _solve_inputs(case, seed)
        systems = [System(*q) for q in _systems(case)]
        s["solver"] = PcgSolver(systems, mode=case["mode"], rtol=RTOL, max_iter=20000, dtau=DTAU)
        s["phi"], s["b"] = phi.to(s["solver"].angle_dtype), b
        if kind == "solve":
            s["phi"] = s["phi"].view(case["nrhs"], -1).requires_grad_()
            s["b"] = b.view(case["nrhs"], -1)
    elif kind == "noise":
        phi, s["eta"] = _noise(case, seed)
        s["boson"] = kernel_to_ref(phi.reshape(1, -1), case["L"], case["Nt"])
        s["est"] = StochaticEstimator(case["L"], case["Nt"], Nrv=case["nrhs"], dtau=DTAU, precision=case["mode"],
                                      cg_rtol=RTOL, noise="z2", autotune=False, corr_dtype=torch.complex64)
    elif kind == "bond":
        phi, eta = _noise(case, seed)
        g = _propagated(eta, case["L"], case["Nt"], _gen(seed, 1))
        s["boson"] = kernel_to_ref(phi.reshape(1, -1), case["L"], case["Nt"])
        s["eta"], s["g"] = eta.to(COMPLEX[case["dtype"]]), g.to(COMPLEX[case["dtype"]])
        s["bb"] = BondBond(case["L"], case["Nt"])
    else:
        s["boson"], s["p0"], s["R"] = _proposal_inputs(case, seed)
        s["hmc"] = HmcSampler(Lx=case["L"], Ltau=case["Nt"], J=1.0, K=1.0, dtau=DTAU, bs=case["chains"], delta_t=0.05,
                              N_leapfrog=case["steps"], precision="mixed", cg_rtol=RTOL, seed=1, autotune=False)
    return s


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "mhm":
        return _C.mhm_vec(s["phi"], s["x"], case["L"], DTAU, 4, 8)
    if kind == "precon":
        return ops.precon_apply(s["x"], s["tau"], case["L"])
    if kind == "force":
        return ops.fermion_force(s["phi"], s["x"], case["L"], DTAU)
    if kind == "solve":
        S = fermion_action(s["phi"], s["b"], s["solver"], case["L"], DTAU)
        return {"S": S.detach(), "grad": torch.autograd.grad(S.sum(), s["phi"])[0]}
    if kind == "batch":
        xi = s["solver"].solve(s["phi"], s["b"]).x.to(torch.complex64)
        out, v = [], 0
        for L, Nt, nrhs, _ in _systems(case):
            n = L * L * Nt * nrhs
            out.append(ops.fermion_force(s["phi"][2 * v:2 * (v + n)].view(nrhs, -1), xi[v:v + n].view(nrhs, -1), L, DTAU))
            v += n
        return out
    if kind == "noise":
        # the correlators take it in the estimator's corr_dtype
        return s["est"].set_eta_G_eta(s["boson"], s["eta"]).to(s["est"].corr_dtype)
    if kind == "bond":
        return s["bb"].get_bond_bond_per_b2(s["eta"], s["g"], s["boson"])
    x, H0, H1, _, _ = s["hmc"].leapfrog_proposer5(s["boson"], p0=s["p0"], R=s["R"])
    return {"x": x, "H0": H0, "H1": H1}


def work(case):
    """Bytes and operations of one pass: for a solve, every iteration's reads
    and writes of its vectors (p, r and x once each way, the operator's result
    once) and of the angles, at about the number of iterations that these fields
    take (more where the pi-flux spectrum's nodes lie on the momentum grid)."""
    kind = case["kind"]
    if kind in ("solve", "batch", "noise", "proposal"):
        systems = _systems(case) if kind != "proposal" else [(case["L"], case["Nt"], case["chains"], False)]
        solves = case["steps"] + 1 if kind == "proposal" else 1
        real = 8 if case.get("mode") == "fp64" else 4
        total = flops = 0
        for L, Nt, nrhs, shared in systems:
            iters, n = (40 + 7.5 * L if L % 4 == 0 else 20 + 5 * L), L * L * Nt
            total += solves * iters * n * real * (14 * nrhs + 2 * (1 if shared else nrhs))
            flops += solves * iters * n * nrhs * 200
        return {"bytes": total, "flops": flops}
    n = case["L"] ** 2 * case["Nt"]
    real = 4 if case["dtype"] == "c64" else 8
    if kind == "bond":
        pairs = case["nrhs"] * (case["nrhs"] - 1) // 2
        # the vectors and the phases; per pair two fields' transforms for three correlators
        return {"bytes": n * 2 * real * (2 * case["nrhs"] + 1),
                "flops": n * pairs * 3 * (40 + 2 * 5 * 2 * math.log2(case["L"]))}
    per = {"mhm": (6, 120), "precon": (4, 52), "force": (6, 270)}[kind]
    return {"bytes": n * case["nvec"] * real * per[0], "flops": n * case["nvec"] * per[1]}


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits
# ---------------------------------------------------------------------------
class _Exact:
    """M, M^dag and the force of angles [n, Nt, L, L, 2], each bond factor as
    c v + s e^{+-i phi} v(partner) over whole slices."""

    def __init__(self, phi, L, n):
        self.L, self.n, self.Nt = L, n, phi.numel() // (2 * L * L * n)
        ang = phi.reshape(n, self.Nt, L * L, 2).double()
        i = torch.arange(L, device=phi.device)
        x, y = (t.reshape(-1) for t in torch.meshgrid(i, i, indexing="xy"))
        up = (x + y) % 2 == 0  # the sites A that the bond groups are counted from
        self.mate, self.origin, self.hop, self.cosh, self.head = [], [], [], [], []
        for g in range(4):
            comp, sign = g % 2, 1 if g < 2 else -1
            d = torch.where(up, sign, -sign)  # A -> its partner, and back
            mate = ((x + d) % L + y * L) if comp == 0 else (x + (y + d) % L * L)
            head = up if sign > 0 else ~up    # the site that its bond starts at
            origin = torch.where(head, x + y * L, mate)
            a = DTAU if g == 0 else DTAU / 2
            ph = torch.polar(torch.full_like(ang[..., 0], math.sinh(a)), ang[..., comp])[..., origin]
            self.hop.append(torch.where(head, ph, ph.conj()))
            self.mate.append(mate)
            self.cosh.append(math.cosh(a))
            self.head.append(head)
        sg = torch.ones(self.Nt, 1, device=phi.device, dtype=torch.float64)
        sg[-1] = -1
        self.sign = sg

    def _F(self, v, g):
        return self.cosh[g] * v + self.hop[g] * v[..., self.mate[g]]

    def _B(self, v):
        for g in (3, 2, 1, 0, 1, 2, 3):
            v = self._F(v, g)
        return v

    def _v(self, v):
        return v.reshape(-1, self.Nt, self.L * self.L).to(torch.complex128)

    def m(self, v):
        w = self._v(v)
        return (w - torch.roll(self.sign * self._B(w), 1, 1)).reshape(v.shape)

    def mh(self, v):
        w = self._v(v)
        return (w - self.sign * self._B(torch.roll(w, -1, 1))).reshape(v.shape)

    def mhm(self, v):
        return self.mh(self.m(v))

    def solve(self, b, tol=1e-14):
        """(M^dag M)^-1 b by CG, restarted from the true residual until it meets tol."""
        x, norm = torch.zeros_like(b), torch.linalg.vector_norm(b, dim=1, keepdim=True)
        for _ in range(4):
            r = b - self.mhm(x)
            if (torch.linalg.vector_norm(r, dim=1, keepdim=True) / norm).max() < tol * 30:
                break
            p, rr, d = r.clone(), (r.abs() ** 2).sum(1, keepdim=True), torch.zeros_like(b)
            for k in range(6000):
                Ap = self.mhm(p)
                al = rr / (p.conj() * Ap).sum(1, keepdim=True).real
                d += al * p
                r = r - al * Ap
                new = (r.abs() ** 2).sum(1, keepdim=True)
                if k % 20 == 0 and (new.sqrt() / norm).max() < tol:
                    break
                p = r + (new / rr) * p
                rr = new
            x = x + d
        return x

    def force(self, xi):
        """-d/dphi of psi^dag (M^dag M)^-1 psi, bond by bond, from its solution xi."""
        w = self._v(xi)
        seq = (3, 2, 1, 0, 1, 2, 3)
        right = [w]
        for g in seq:
            right.append(self._F(right[-1], g))
        left = right[-1] - self.sign * torch.roll(w, -1, 1)
        F = torch.zeros((self.n, self.Nt, self.L * self.L, 2), device=w.device, dtype=torch.float64)
        for k, g in enumerate(seq):
            R, mate, h = right[6 - k], self.mate[g], self.head[g]
            hop = 1j * self.hop[g]  # d/dphi of the hop out of the bond's first site
            t = 2 * (left.conj() * hop * R[..., mate] + left[..., mate].conj() * hop.conj() * R).real
            F[..., g % 2] += torch.where(h, t, torch.zeros_like(t))
            left = self._F(left, g)
        return F.reshape(self.n, -1)


def _exact_bond(eta, g, boson, L, Nt):
    n = eta.shape[0]
    ec, g = eta.conj().reshape(n, Nt, L, L), g.reshape(n, Nt, L, L)
    e = torch.polar(torch.ones((Nt, L, L), device=g.device, dtype=torch.float64), boson[0, 0].permute(2, 1, 0).double())
    sx = lambda v: torch.roll(v, -1, -1)  # noqa: E731  v(r + x)
    corr = lambda a, b: (torch.fft.ifft2(a, norm="forward") * torch.fft.fft2(b)).sum((0, 1))  # noqa: E731
    T1 = torch.zeros((L, L), device=g.device, dtype=torch.complex128)
    T21, T4 = T1.clone(), T1.clone()
    for s in range(n - 1):
        es, gs, et, gt = ec[s], g[s], ec[s + 1:], g[s + 1:]
        T1 += corr(es * sx(gt) * e, sx(gs) * et * e)
        T4 += corr(sx(es) * gt * e.conj(), gs * sx(et) * e.conj())
        T21 += corr((sx(es) * gt + sx(et) * gs) * e.conj() / 2, (sx(gs) * et + sx(gt) * es) * e / 2)
    back = lambda S, m: torch.fft.ifft2(S, norm="forward") / (m * Nt * float(L) ** 4)  # noqa: E731
    pairs = n * (n - 1) // 2
    T1, T21, T4 = -back(T1, pairs), -back(T21, pairs), -back(T4, pairs)
    bx = lambda v: torch.roll(v, 1, -1)  # noqa: E731  v(r - x)
    T1[0, -1] += (sx(g) * bx(ec) * e * bx(e)).mean()
    T21[0, 0] += (g * ec).mean()
    T4[0, 1] += (g * sx(sx(ec)) * (e * sx(e)).conj()).mean()
    v = sx(g) * ec * e + g * sx(ec) * e.conj()
    T = T1 + T21 + torch.roll(torch.flip(T21, (0, 1)), (1, 1), (0, 1)) + T4
    BB = 2 * T + 4 * back(corr(v, v), n)
    BBk = torch.roll(torch.fft.ifft2(BB, norm="forward"), (L // 2, L // 2), (0, 1))
    return {"BB0_r": 2 * T.real, "BB_r": BB.real, "B_r": v.mean((0, 1)).real, "BB_k": BBk.real}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mhm", "force"):
        s = prepare(case, seed)
        E = _Exact(s["phi"], case["L"], case["nvec"])
        x = s["x"].to(torch.complex128)
        return E.mhm(x) if kind == "mhm" else E.force(x)
    if kind == "precon":
        s = prepare(case, seed)
        rp, col, val = s["tau"]
        P = torch.sparse_csr_tensor(rp, col, val, (case["Nt"], case["Nt"])).to_dense().to(torch.complex128)
        return (P @ s["x"].to(torch.complex128).view(case["nvec"], case["Nt"], -1)).reshape(s["x"].shape)
    if kind in ("solve", "batch"):
        phi, b = _solve_inputs(case, seed)
        out, v = [], 0
        for L, Nt, nrhs, _ in _systems(case):
            n = L * L * Nt * nrhs
            E, psi = _Exact(phi[2 * v:2 * (v + n)], L, nrhs), b[v:v + n].view(nrhs, -1)
            xi = E.solve(psi)
            out.append(E.force(xi))
            v += n
        return {"S": (psi.conj() * xi).sum(1).real, "grad": -out[0]} if kind == "solve" else out
    if kind == "noise":
        if case["nrhs"] * case["L"] ** 3 * case["Nt"] > 1e8:
            return None
        phi, eta = _noise(case, seed)
        E = _Exact(phi, case["L"], 1)
        return E.solve(E.mh(eta))
    if kind == "bond":
        s = prepare(case, seed)
        return _exact_bond(s["eta"].to(torch.complex128), s["g"].to(torch.complex128), s["boson"], case["L"], case["Nt"])
    # a proposal integrates in single precision: no value of its own in 64 bits
    return None
