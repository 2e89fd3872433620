"""Timed workloads of the B200 NEGF solvers.

Every case is one call sequence that a program makes through the public entry points:

  solve    Solver.solve_scf (fresh start) + current + observables: one IV point of QUICHOTTE.
           Orders 0, 1 and 2, the FP64 and the mixed form. `steps` is the reference's maxscf
           key; the non-mixed solves stop there, so every seed does the same work. It is small
           where the history is kept in single precision: rounding a pair to FP32 makes the
           path of a longer solve depend on the last bits of its residuals.
  residual Solver.residual on host arrays: one evaluation of the SCF function, as a program
           with a mixing scheme of its own calls it.
  sancho   SanchoSolver.solve_scf + current + observables: one IV point of SANCHO.
  inverse  qs_invert_batched_noalloc on device arrays: the Dyson inversion for a program that
           owns its device memory.

The models are the benchmark's helices and chains (wide-band leads, Gamma = 0.5 eV, t = 1 eV,
lambda = 0.01 eV) with a weak random on-site disorder, a random voltage and a random U near
the stated one, all drawn from the seed.

    listed()              the cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   the handle and inputs that a program keeps
    run(state)            one pass, its outputs
    work(case)            bytes and flops that the pass cannot do without
    exact(case, seed)     the outputs in plain 64-bit torch, where that is quick enough
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "quichotte-and-sancho_b200")
KB = 8.6173303e-5  # eV/K, the reference's Boltzmann constant
PITCH, RADIUS = 0.34, 0.7  # nm per turn, nm


def _solve(name, ions, turns, n, order, steps, nhist=8, U=1.0, alpha=0.5, single=True, mixed=False, tolf=1e-6):
    return dict(name=name, kind="solve", ions=ions, turns=turns, n=n, order=order, steps=steps, nhist=nhist, U=U,
                alpha=alpha, single=single, mixed=mixed, tolf=tolf)


def listed():
    return [
        # a non-interacting transmission scan: the benchmark's helix and grid at order 0
        _solve("order0_scan", 10, 6, 16384, 0, 1, U=0.0),
        # Hartree-Fock on an odd grid
        _solve("order1_hartree_fock", 8, 3, 4001, 1, 5, U=0.3, alpha=0.3, single=False),
        # the regression suite's smallest order-2 model: launches and latency
        _solve("order2_smallest", 4, 1, 329, 2, 6, U=0.8),
        # the CPU-runnable configuration of the benchmark (16 states, 4096 energies, mixing 0.1)
        _solve("order2_small", 4, 2, 4096, 2, 6, nhist=16, U=0.5, alpha=0.1, tolf=1e-8),
        # a grid as the energy-step keys give it, neither a power of two nor a round number; a
        # double-precision history that fills up
        _solve("order2_odd_grid", 5, 4, 5003, 2, 10, single=False),
        # the largest grid of the serving stream on one of its small molecules
        _solve("order2_fine_grid", 4, 3, 32768, 2, 5, U=0.6),
        # the benchmark's 120 x 120 helix with its 16-column history, a quarter of its grid
        _solve("order2_large", 10, 6, 4096, 2, 5, nhist=16),
        # the widest molecule of the serving stream (192 states)
        _solve("order2_widest", 12, 8, 1201, 2, 4, nhist=4, U=0.5),
        # the mixed-precision form, converged
        _solve("order2_mixed", 5, 2, 6001, 2, 80, U=0.5, single=False, mixed=True, tolf=1e-10),
        # one SCF function evaluation through host arrays
        dict(name="residual_host", kind="residual", ions=4, turns=2, n=1021, U=0.5),
        # SANCHO's order-3 chain of the benchmark
        dict(name="sancho_order3", kind="sancho", sites=10, n=883, order=3, steps=8, U=0.5),
        # the benchmark's matrix order through the allocation-free inversion
        dict(name="inverse_device", kind="inverse", N=120, batch=1024),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: molecules from 4 to 96 sites, grids from 300 to 20000 energies (any
    integer, and the serving stream's powers of two), every order and form."""
    limit = _cost(next(c for c in listed() if c["name"] == "order2_large"))
    kind = rng.choices(["order2", "order01", "mixed", "residual", "sancho", "inverse"], [6, 2, 1, 1, 2, 2])[0]
    if kind == "inverse":
        N = _logint(rng, 8, 256)
        return dict(kind="inverse", N=N, batch=_logint(rng, 64, max(65, min(16384, int(2e7 / N ** 2)))))
    if kind == "sancho":
        c = dict(kind="sancho", sites=rng.randint(3, 14), n=_logint(rng, 200, 2000), order=rng.choice([2, 3, 3]),
                 steps=rng.randint(5, 10), U=round(rng.uniform(0.2, 0.8), 3))
        while c["sites"] ** 2 * c["n"] ** 2 * c["steps"] > 2e9:
            c["n"] = int(c["n"] * 0.8)
        return c
    n = rng.choice([1024, 2048, 4096, 8192, 16384]) if rng.random() < 0.35 else _logint(rng, 300, 20000)
    if kind == "residual":
        return dict(kind="residual", ions=rng.randint(3, 6), turns=rng.randint(1, 2), n=min(n, _logint(rng, 300, 3000)),
                    U=round(rng.uniform(0.2, 1.0), 3))
    single = rng.random() < 0.6
    c = _solve("", rng.randint(3, 12), rng.randint(1, 8), n, 2, rng.randint(3, 5) if single else rng.randint(5, 10),
               nhist=rng.choice([4, 8, 16]), U=round(rng.uniform(0.2, 0.8), 3), alpha=rng.choice([0.3, 0.5]),
               single=single)
    del c["name"]
    if kind == "order01":
        c.update(order=rng.choice([0, 1]), nhist=8, alpha=0.3, U=round(rng.uniform(0.15, 0.3), 3), single=False,
                 steps=rng.randint(3, 5))
        if c["order"] == 1:  # a long chain's Hartree-Fock levels are too sharp to be reproducible
            c.update(ions=rng.randint(3, 8), turns=rng.randint(1, 2), n=min(n, 6000))
    if kind == "mixed":
        # small enough to converge from a fresh start at every seed
        c.update(ions=rng.randint(3, 5), turns=rng.randint(1, 2), steps=80, single=False, mixed=True, tolf=1e-10, U=0.5,
                 alpha=0.5, nhist=8, n=_logint(rng, 4096, 16384))
    while _cost(c) > limit and c["n"] > 600:
        c["n"] = max(600, int(c["n"] * 0.8))
    while _cost(c) > limit and c["turns"] > 1:
        c["turns"] -= 1
    return c


# ---------------------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------------------
def _cost(c):
    """Seconds of a pass at 6.5 TB/s and 37 TFLOP/s of FP64, to compare cases by size."""
    w = work(c)
    return w["bytes"] / 6.5e12 + w["flops"] / 37e12


def work(c):
    if c["kind"] == "inverse":
        return {"bytes": 32.0 * c["N"] ** 2 * c["batch"], "flops": 8.0 * c["N"] ** 3 * c["batch"]}
    if c["kind"] == "sancho":
        Na, n = c["sites"], c["n"]
        L = 2 * n
        k = c["steps"]
        fft = 5.0 * L * math.log2(L) * Na * Na
        per = n * 24.0 * Na ** 3 + fft * (10 if c["order"] == 2 else 26)
        if c["order"] == 3:
            per += 2 * L * 40.0 * Na ** 3
        nv = 3.0 * Na * Na * n
        return {"bytes": 8.0 * nv * (8 * k + sum(2 * min(s, 8) + 2 for s in range(k))), "flops": per * k}
    N, n = 2 * c["ions"] * c["turns"], c["n"]
    nv = 3.0 * N * N * n
    Nf = 2.0 * n
    fft = 3.0 * N * N * 5.0 * Nf * math.log2(Nf)
    if c["kind"] == "residual":
        return {"bytes": 16.0 * nv, "flops": 20.0 * n * N ** 3 + fft}
    if c["order"] < 2:
        k = 1 if c["order"] == 0 else c["steps"] + 2
        return {"bytes": 8.0 * n * (N + 2) + 32.0 * N * N, "flops": 8.0 * n * N ** 3 * k}
    k = 20 if c["mixed"] else c["steps"]  # a mixed solve converges in about 20 steps
    el = 4.0 if c["single"] else 8.0
    hist = sum(el * nv * (2 * min(s, c["nhist"]) + 2) for s in range(k))
    return {"bytes": 8.0 * nv * 8 * k + hist + 8.0 * n * (N + 2), "flops": (k + 1) * 20.0 * n * N ** 3 + k * fft}


# ---------------------------------------------------------------------------------------
# models
# ---------------------------------------------------------------------------------------
class _Grid:
    """The arrays of a model: H, lead matrices, U, energies, and the scalars of its input."""


def _helix_H(ions, turns):
    """The reference's helix Hamiltonian (spin fastest): nearest-neighbour hopping t = 1 eV and
    second-neighbour spin-orbit hopping of strength lambda = 0.01 eV."""
    ns = ions * turns
    length = PITCH * turns * (ions - 1) / ions
    i = np.arange(ns)
    ang = i * 2 * np.pi / ions
    pos = np.stack([RADIUS * np.cos(ang), RADIUS * np.sin(ang), length * i / (turns * (ions - 1))], axis=1)
    H = np.zeros((2 * ns, 2 * ns), np.complex128)
    for s in range(ns):
        if s + 1 < ns:
            H[2 * s, 2 * s + 2] = H[2 * s + 1, 2 * s + 3] = 1.0
        if s + 2 < ns:
            d1, d2 = pos[s] - pos[s + 1], pos[s] - pos[s + 2]
            v = np.cross(d1 / np.linalg.norm(d1), d2 / np.linalg.norm(d2))
            sx = np.array([[v[2], v[0] - 1j * v[1]], [v[0] + 1j * v[1], -v[2]]])
            H[2 * s:2 * s + 2, 2 * s + 4:2 * s + 6] = 0.01j * sx
    return H + np.conj(H).T


def _helix(c, seed):
    rng = np.random.default_rng(seed)
    g = _Grid()
    ns = c["ions"] * c["turns"]
    g.N, g.n, g.order = 2 * ns, c["n"], c.get("order", 2)
    dis = 0.05 * rng.standard_normal(ns)
    g.H = _helix_H(c["ions"], c["turns"]) + np.diag(np.repeat(dis, 2))
    g.GammaL = np.zeros((g.N, g.N), np.complex128)
    g.GammaR = np.zeros_like(g.GammaL)
    g.GammaL[0, 0] = g.GammaL[1, 1] = 0.5
    g.GammaR[-2, -2] = g.GammaR[-1, -1] = 0.5
    g.U = np.zeros(g.N)
    g.U[0::2] = c["U"] * (1.0 + 0.02 * rng.standard_normal())
    g.V = -0.8 + 0.1 * rng.random()
    g.mu, g.beta = 0.0, 1.0 / (KB * 300.0)
    half = 10.0 if c["n"] >= 1500 else 4.0  # coarse grids span less
    g.delta = 2 * half / c["n"]
    g.omega = -half + g.delta * np.arange(1, c["n"] + 1)
    return g


def _qb():
    if PKG not in sys.path:
        sys.path.insert(0, PKG)
    import quichotte_b200
    return quichotte_b200


def _solver(c, g):
    qb = _qb()
    turns, ions = c["turns"], c["ions"]
    m = qb.Model.helix(N_ions=ions, N_turns=turns, hel_length=PITCH * turns * (ions - 1) / ions, hel_radius=RADIUS,
                       hand=1.0, E_CC=0.0, t_hop=1.0, lamb=0.01, U_int=1.0, GammaL_up=0.5, GammaL_down=0.5, GammaR=0.5,
                       T=300.0, mu=0.0, dw=1.0, up=1.0, delta=0.5, order=g.order)
    m.H, m.U_site, m.GammaL, m.GammaR = g.H, g.U, g.GammaL, g.GammaR
    m.omega, m.n_omega, m.delta, m.mu, m.beta = g.omega, g.n, g.delta, g.mu, g.beta
    prec = qb.QS_PREC_MIXED if c.get("mixed") else qb.QS_PREC_FP64
    return qb.Solver(m, precision=prec, alpha_mix=c.get("alpha", 0.5), nhist=c.get("nhist", 8),
                     maxscf=c.get("steps", 8), tolf=c.get("tolf", 1e-6), tolf_order1=1e-12,
                     single_history=int(c.get("single", True)))


def _chain(c, seed):
    rng = np.random.default_rng(seed)
    g = _Grid()
    g.N, g.n, g.order = c["sites"], c["n"], c["order"]
    g.H = np.zeros((g.N, g.N), np.complex128)
    for s in range(g.N - 1):
        g.H[s, s + 1] = g.H[s + 1, s] = -0.4
    g.H += np.diag(2.0 + 0.03 * rng.standard_normal(g.N))
    g.GammaL = np.zeros((g.N, g.N), np.complex128)
    g.GammaR = np.zeros_like(g.GammaL)
    g.GammaL[0, 0] = g.GammaR[-1, -1] = 1.0
    g.U = np.full(g.N, c["U"] * (1.0 + 0.02 * rng.standard_normal()))
    g.V = -0.5 + 0.1 * rng.random()
    g.mu, g.beta = 2.0, 1.0 / (KB * 300.0)
    lo, hi = 0.0, 4.0
    g.delta = (hi - lo) / c["n"]
    g.omega = lo + g.delta * np.arange(1, c["n"] + 1)
    return g


def _sancho_solver(c, g):
    _qb()
    import sancho_b200 as sb
    with tempfile.TemporaryDirectory(prefix="sancho_case_") as d:
        with open(os.path.join(d, "input.dat"), "w") as f:
            f.write(f"T = 300.0\nV = -0.5\nVf = 0.5\ndelv = 0.25\nmu = 2.0\nN_sites = {g.N}\nE_CC = 2.0\nt_hop = -0.4\n"
                    f"U_int = 0.5\norder = {g.order}\ndw = 1.0\nup = 1.0\ndelta = 0.1\nalpha_mix = 0.3\nnhist = 8\n"
                    "maxscf = 200\ntolf = 1.d-6\nGammaL = 1.0\nGammaR = 1.0\n")
        m = sb.SanchoModel.load(d)
    m.H, m.U_site, m.GammaL, m.GammaR = g.H, g.U, g.GammaL, g.GammaR
    m.omega, m.n_omega, m.delta, m.mu, m.beta = g.omega, g.n, g.delta, g.mu, g.beta
    return sb.SanchoSolver(m, alpha_mix=0.3, nhist=8, maxscf=c["steps"], tolf=1e-12)


def _matrices(c, seed):
    """Dyson matrices w - H - Sigma of one random Hamiltonian: a Hermitian H with its spectrum
    in about [-2, 2], energies over it, and a damping between 0.05 and 0.5 on each state."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    N, b = c["N"], c["batch"]
    r = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda", generator=gen)
    H = torch.complex(r(N, N), r(N, N)) / math.sqrt(2 * N)
    H = (H + H.mH) / math.sqrt(2.0)
    w = torch.linspace(-3.0, 3.0, b, dtype=torch.float64, device="cuda")
    damp = 0.05 + 0.45 * torch.rand(b, N, dtype=torch.float64, device="cuda", generator=gen)
    return torch.diag_embed(torch.complex(w[:, None].expand(b, N).contiguous(), damp)) - H


# ---------------------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------------------
def prepare(c, seed):
    if c["kind"] == "inverse":
        qb = _qb()
        # the kernel sees the rows of a torch matrix as columns: it inverts the transposes in place
        return dict(kind="inverse", lib=qb._lib, A=_matrices(c, seed).contiguous(), N=c["N"], batch=c["batch"],
                    info=torch.zeros(c["batch"], dtype=torch.int32, device="cuda"))
    if c["kind"] == "sancho":
        g = _chain(c, seed)
        return dict(kind="sancho", solver=_sancho_solver(c, g), V=g.V)
    g = _helix(c, seed)
    s = dict(kind=c["kind"], solver=_solver(c, g), V=g.V, mixed=bool(c.get("mixed")))
    if c["kind"] == "residual":
        s["x"] = _noisy_start(g, seed)
    return s


def run(s):
    if s["kind"] == "inverse":
        X = s["A"].clone()
        rc = s["lib"].qs_invert_batched_noalloc(s["N"], s["batch"], X.data_ptr(), s["info"].data_ptr(),
                                                torch.cuda.current_stream().cuda_stream)
        if rc != 0:
            raise RuntimeError(f"qs_invert_batched_noalloc: {rc}")
        return dict(inverse=X, info=s["info"])
    sol = s["solver"]
    if s["kind"] == "residual":
        F, abort = sol.residual(s["V"], s["x"])
        return dict(F=F, abort=abort)
    r = sol.solve_scf(s["V"], True)
    J = sol.current(s["V"])
    out = dict(sol.observables(), current=np.atleast_1d(np.array(J)), converged=r["converged"])
    if not s.get("mixed"):  # the step at which a mixed solve converges is not a result
        out["n_iter"] = r["n_iter"]
    return out


# ---------------------------------------------------------------------------------------
# the same results in plain 64-bit torch
# ---------------------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Exact:
    """QUICHOTTE's equations on full (n, N, N) complex128 tensors."""

    def __init__(self, g):
        dev = _dev()
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
        self.g, self.N, self.n = g, g.N, g.n
        self.GL, self.GR, self.U, self.w = t(g.GammaL), t(g.GammaR), t(g.U), t(g.omega)
        self.Hemb = -t(g.H) + 0.5j * (self.GL + self.GR)
        f = lambda V: 1.0 / (torch.exp(torch.clamp((self.w - g.mu + V) * g.beta, max=700.0)) + 1.0)
        self.fL, self.fR = f(g.V)[:, None, None], f(0.0)[:, None, None]
        self.pp = g.delta / (2 * math.pi)
        self.iu = torch.triu_indices(g.N, g.N, 1, device=dev)

    def gr(self, Sig1=None, SR=None):
        W = torch.zeros(self.n, self.N, self.N, dtype=torch.complex128, device=self.w.device)
        W += self.Hemb if Sig1 is None else self.Hemb - Sig1
        if SR is not None:
            W -= SR
        W.diagonal(dim1=1, dim2=2).add_(self.w[:, None])
        out = torch.empty_like(W)
        for k in range(0, self.n, 2048):
            out[k:k + 2048] = torch.linalg.inv(W[k:k + 2048])
        return out

    def glesser(self, Gr, SL=None):
        S = 1j * (self.fL * self.GL + self.fR * self.GR)
        if SL is not None:
            S = S + SL
        return Gr @ S @ Gr.mH

    def pack(self, Gr, Gl):
        u = Gl[:, self.iu[0], self.iu[1]]
        d = Gl.diagonal(dim1=1, dim2=2).imag
        return torch.cat([torch.view_as_real(Gr).reshape(-1), torch.view_as_real(u).reshape(-1), d.reshape(-1)])

    def unpack(self, x):
        n, N = self.n, self.N
        a, b = 2 * n * N * N, n * N * (N - 1)
        Gr = torch.view_as_complex(x[:a].reshape(n, N, N, 2).contiguous())
        u = torch.view_as_complex(x[a:a + b].reshape(n, -1, 2).contiguous())
        Gl = torch.zeros_like(Gr)
        Gl[:, self.iu[0], self.iu[1]] = u
        Gl = Gl - Gl.mH
        Gl.diagonal(dim1=1, dim2=2).add_(1j * x[a + b:].reshape(n, N))
        return Gr, Gl

    def onsite(self, M):
        """The 2x2 on-site blocks of a matrix, zero elsewhere."""
        i = torch.arange(self.N, device=M.device) // 2
        return M * (i[:, None] == i[None, :])

    def sigma1(self, Gt0):
        """First order from the equal-time G^<: i U (G - tr G) on every on-site block."""
        s = self.N // 2
        i = torch.arange(s, device=Gt0.device)
        B = Gt0.reshape(s, 2, s, 2)[i, :, i, :]
        tr = B.diagonal(dim1=1, dim2=2).sum(-1)
        T = B - tr[:, None, None] * torch.eye(2, dtype=B.dtype, device=B.device)
        out = torch.zeros_like(Gt0)
        out.view(s, 2, s, 2)[i, :, i, :] = 1j * self.U[0::2][:, None, None] * T
        return out

    def sigma2(self, Gr, Gl):
        n, N, s = self.n, self.N, self.N // 2
        Nf = 2 * n
        F = lambda G: torch.fft.fft(G.permute(1, 2, 0).contiguous(), Nf, dim=2).view(s, 2, s, 2, Nf)
        R, L = F(Gr), F(Gl)
        neg = (-torch.arange(Nf, device=R.device)) % Nf
        comp = lambda M: [[M[:, a, :, b] for b in (0, 1)] for a in (0, 1)]
        part = lambda M: [[M[:, a, :, b].transpose(0, 1)[..., neg] for b in (0, 1)] for a in (0, 1)]
        r, l, rp, lp = comp(R), comp(L), part(R), part(L)
        two = range(2)
        dag = lambda X: [[X[b][a].conj() for b in two] for a in two]
        mm = lambda X, Y: [[X[a][0] * Y[0][b] + X[a][1] * Y[1][b] for b in two] for a in two]
        add = lambda X, Y, q=1: [[X[a][b] + q * Y[a][b] for b in two] for a in two]
        adj = lambda M: [[M[1][1], -M[0][1]], [-M[1][0], M[0][0]]]
        a_ij, a_ji = dag(rp), dag(r)
        G_ij, G_ji = add(add(l, r), a_ij, -1), add(add(lp, rp), a_ji, -1)
        sL = mm(l, adj(mm(G_ji, l)))
        sR = add(mm(r, adj(mm(lp, G_ij))), mm(l, adj(add(mm(lp, r), mm(a_ji, l)))))
        c = self.pp ** 2 * self.U[0::2][:, None] * self.U[0::2][None, :]

        def back(S):
            out = torch.empty(n, s, 2, s, 2, dtype=torch.complex128, device=R.device)
            for a in two:
                for b in two:
                    out[:, :, a, :, b] = (torch.fft.ifft(S[a][b], dim=2)[..., :n] * c[:, :, None]).permute(2, 0, 1)
            return out.view(n, N, N)
        return back(sR), back(sL)

    def residual(self, x):
        """The packed G_out[x] - x, and the self-energies of x."""
        Gr, Gl = self.unpack(x)
        S1 = self.sigma1(self.onsite(Gl.sum(0) * self.pp))
        SR, SL = self.sigma2(Gr, Gl)
        G = self.gr(S1, SR)
        return self.pack(G, self.glesser(G, SL)) - x, (S1, SR, SL)

    def observables(self, sig):
        S1, SR, SL = sig
        G = self.gr(S1, SR)
        Gl = self.glesser(G, SL)
        X = (self.fL - 1.0) * Gl - self.fL * (Gl + G - G.mH)
        t = (1j * self.GL * X.transpose(1, 2)).sum(2).real / (2 * math.pi)
        trU, trD = t[:, 0::2].sum(1), t[:, 1::2].sum(1)
        return dict(G_less_obs=self.onsite(Gl.sum(0) * self.pp), dosd=G.diagonal(dim1=1, dim2=2).imag.mT,
                    trU=trU, trD=trD, current=torch.stack([trU.sum(), trD.sum()]) * self.g.delta)


def _broyden(residual, x, alpha, nhist, maxscf, tolf, single):
    """Johnson's modified Broyden mixing as the reference does it; returns the result of the
    last residual(x) -> (F, extra), its extra and the step count."""
    dt = torch.float32 if single else torch.float64
    dF, Uc, stored = [], [], 0
    F0 = x0 = None
    for its in range(1, maxscf + 1):
        F, extra = residual(x)
        if float(F.abs().max()) < tolf:
            return x, extra, its, True
        if F0 is not None and nhist > 0:
            fn = float(torch.linalg.vector_norm(F - F0))
            if fn > 0.0:
                d = (F - F0) / fn
                u = alpha * d + (x - x0) / fn
                if len(dF) < nhist:
                    dF.append(d.to(dt))
                    Uc.append(u.to(dt))
                else:
                    dF[stored % nhist], Uc[stored % nhist] = d.to(dt), u.to(dt)
                stored += 1
                del d, u
        new = x + alpha * F
        if dF:
            k = len(dF)
            A = torch.zeros(k, k, dtype=torch.float64)
            b = torch.zeros(k, dtype=torch.float64)
            for i in range(k):
                di = dF[i].double()
                b[i] = torch.dot(di, F).item()
                for j in range(i, k):
                    A[i, j] = A[j, i] = torch.dot(di, dF[j].double()).item()
            gam = torch.linalg.solve(A + 1e-4 * torch.eye(k, dtype=torch.float64), b)
            for i in range(k):
                new -= float(gam[i]) * Uc[i].double()
        F0, x0, x = F, x, new
    return x0, extra, maxscf, False


def _fresh(ex):
    G = ex.gr()
    return G, ex.glesser(G)


def _ref_layout(ex, Gr, Gl):
    """pack_gf's block per energy: Re G^r, Im G^r (row-major), Re of the strict upper triangle
    of G^<, Im of its upper triangle."""
    n = ex.n
    full = torch.triu_indices(ex.N, ex.N, 0, device=Gr.device)
    return torch.cat([Gr.real.reshape(n, -1), Gr.imag.reshape(n, -1), Gl[:, ex.iu[0], ex.iu[1]].real,
                      Gl[:, full[0], full[1]].imag], dim=1).reshape(-1)


def _noisy_start(g, seed):
    """A host SCF vector near the fresh start: the non-interacting G plus noise."""
    ex = _Exact(g)
    x = _ref_layout(ex, *_fresh(ex)).cpu().numpy()
    return x + 1e-3 * np.random.default_rng(seed + 1).standard_normal(x.size)


def _from_ref_layout(ex, x):
    n, N = ex.n, ex.N
    b = torch.as_tensor(x, device=ex.w.device).reshape(n, -1)
    nf, nsu = N * N, N * (N - 1) // 2
    Gr = torch.complex(b[:, :nf], b[:, nf:2 * nf]).reshape(n, N, N)
    full = torch.triu_indices(N, N, 0, device=b.device)
    up = torch.zeros(n, N, N, dtype=torch.complex128, device=b.device)
    up[:, full[0], full[1]] = 1j * b[:, 2 * nf + nsu:]
    up[:, ex.iu[0], ex.iu[1]] += b[:, 2 * nf:2 * nf + nsu]
    strict = up.triu(1)
    return Gr, up - strict.mH


def _exact_solve(c, seed):
    g = _helix(c, seed)
    ex = _Exact(g)
    if g.order == 0:
        o, its, conv = ex.observables((None, None, None)), 1, True
    elif g.order == 1:
        s = g.N // 2
        i = torch.arange(s, device=ex.w.device)
        blocks = lambda M: torch.view_as_real(M.reshape(s, 2, s, 2)[i, :, i, :].contiguous()).reshape(-1)

        def full(x):
            M = torch.zeros(g.N, g.N, dtype=torch.complex128, device=x.device)
            M.view(s, 2, s, 2)[i, :, i, :] = torch.view_as_complex(x.reshape(s, 2, 2, 2).contiguous())
            return M

        def res(x):
            S1 = ex.sigma1(full(x))
            return blocks(ex.glesser(ex.gr(S1)).sum(0) * ex.pp) - x, S1
        x0 = blocks(_fresh(ex)[1].sum(0) * ex.pp)
        _, S1, its, conv = _broyden(res, x0, c["alpha"], c["nhist"], c["steps"], 1e-12, c["single"])
        o = ex.observables((S1, None, None))
    else:
        _, sig, its, conv = _broyden(ex.residual, ex.pack(*_fresh(ex)), c["alpha"], c["nhist"], c["steps"], c["tolf"],
                                     c["single"])
        o = ex.observables(sig)
    o = {k: v.cpu().numpy() for k, v in o.items()}
    o["converged"] = conv
    if not c["mixed"]:
        o["n_iter"] = its
    return o


def _exact_sancho(c, seed):
    g = _chain(c, seed)
    ex = _Exact(g)  # its fermi functions, G^r and pack are SANCHO's too
    n, Na, pp = g.n, g.N, ex.pp
    L = 4 * n
    U = ex.U.to(torch.complex128)
    f = lambda A: torch.fft.fft(A, L, dim=0)
    fi = lambda A: torch.fft.ifft(A, dim=0)
    corr = lambda A, B: fi(f(A) * f(B.conj()).conj())  # sum_k A(k) B(k - m) at m mod L

    def self_energies(Gr, Gl):
        Ga, Gg = Gr.mH, Gl + Gr - Gr.mH
        ch = lambda A, B: torch.roll(corr(A, B.transpose(1, 2)), n - 1, 0)[:2 * n - 1] * pp  # m = -(n-1) .. n-1
        chi = dict(g=ch(Gg, Gl), l=ch(Gl, Gg), r=ch(Gr, Gl) + ch(Gl, Ga), a=ch(Ga, Gl) + ch(Gl, Gr))

        def conv(E, X):  # sum_k E(k) X(w - k)
            return fi(f(E) * f(X))[n - 1:2 * n - 1]
        cu = pp * U[:, None] * U[None, :]
        SR, SL = cu * (conv(Gr, chi["g"]) + conv(Gl, chi["r"])), cu * conv(Gl, chi["l"])
        if g.order == 3:
            ph = lambda A, B: fi(f(A) * f(B))[:2 * n - 1] * pp
            phi = dict(g=ph(Gg, Gg), l=ph(Gl, Gl), r=ph(Gr, Gg) + ph(Gl, Gr), a=ph(Ga, Gg) + ph(Gl, Ga))
            prod = lambda Y: dict(g=(Y["r"] * U) @ Y["g"] + (Y["g"] * U) @ Y["a"],
                                  l=(Y["r"] * U) @ Y["l"] + (Y["l"] * U) @ Y["a"], r=(Y["r"] * U) @ Y["r"])
            D, P = prod(chi), prod(phi)
            T = lambda E: E.transpose(1, 2)
            pc = lambda E, X: fi(f(E.conj()).conj() * f(X))[:n]  # sum_k E(k) X(w + k)
            SR = SR + 1j * cu * (conv(Gr, D["g"]) + conv(Gl, D["r"]) + pc(T(Ga), P["g"]) + pc(T(Gg), P["r"]))
            SL = SL + 1j * cu * (conv(Gl, D["l"]) + pc(T(Gg), P["l"]))
        return SR, SL

    def res(x):
        Gr, Gl = ex.unpack(x)
        t0 = Gl.diagonal(dim1=1, dim2=2).sum(0) * pp
        SR, SL = self_energies(Gr, Gl) if g.order >= 2 else (None, None)
        G = ex.gr(torch.diag(-1j * U * t0), SR)
        return ex.pack(G, ex.glesser(G, SL)) - x, t0
    x, t0, its, conv = _broyden(res, ex.pack(*_fresh(ex)), 0.3, 8, c["steps"], 1e-12, False)
    Gr, Gl = ex.unpack(x)
    X = (ex.fL - 1.0) * Gl - ex.fL * (Gl + Gr - Gr.mH)
    J = 2.0 * g.delta * ((1j * ex.GL * X.transpose(1, 2)).sum((1, 2)).real / (2 * math.pi)).sum()
    return dict(G_less_t0=t0.cpu().numpy(), spectral=(-2.0 * Gr.diagonal(dim1=1, dim2=2).imag).mT.cpu().numpy(),
                current=np.array([float(J)]), converged=conv, n_iter=its)


def exact(c, seed):
    if c["kind"] == "inverse":
        return dict(inverse=torch.linalg.inv(_matrices(c, seed)), info=None)
    if not torch.cuda.is_available() and work(c)["flops"] > 2e11:
        return None
    if c["kind"] == "sancho":
        return _exact_sancho(c, seed)
    if c["kind"] == "residual":
        g = _helix(c, seed)
        ex = _Exact(g)
        x = _noisy_start(g, seed)
        Gr, Gl = _from_ref_layout(ex, x)
        S1 = ex.sigma1(ex.onsite(Gl.sum(0) * ex.pp))
        SR, SL = ex.sigma2(Gr, Gl)
        G = ex.gr(S1, SR)
        F = _ref_layout(ex, G, ex.glesser(G, SL)).cpu().numpy() - x
        return dict(F=F, abort=False)
    return _exact_solve(c, seed)
