"""Performance cases of the walker step, the local energies and their derivatives.

Each case is one call (or one driver block) through the package's public classes on a seeded
synthetic Hamiltonian.  Kinds:

``block``     ten steps of the driver loop (``AFQMC.step``) in the throughput mode: fields and
              population control on the device, steps replayed from CUDA graphs, reortho and
              population control every 5 steps, the local energy at the block's end;
``step``      one ``PhaselessGeneric.propagate_walkers`` with caller-supplied fields (reortho and
              population control every 5th pass);
``greens``    ``SingleDet.calc_greens_function``;
``reortho``   ``UHFWalkers.reortho``;
``energy``    the local energies of a walker batch;
``gradient``  local energies and their gradient with respect to the half-rotated Green's functions
              (``LocalEnergyGreens``, forward and backward).

Sizes: W walkers, M basis functions, na + nb electrons, X Cholesky vectors.  ``trial`` is "rhf"
(identical spin blocks, computed once, as the driver does), "uhf", or "complex" (UHF trial with
complex Cholesky vectors).
"""
import itertools
import math

import numpy as np
import torch

DT = 0.005
STEPS = 10  # steps of a block
EVERY = 5  # steps between reorthogonalisations and population controls


def _case(name, kind, W, M, na, nb, X, trial, precision="fp64"):
    return dict(name=name, kind=kind, W=W, M=M, na=na, nb=nb, X=X, trial=trial, precision=precision)


def listed():
    return [
        # the smallest run: a first-row molecule in a small basis, 64 walkers -- latency and launches
        _case("block_fp64_w64_m26", "block", 64, 26, 5, 5, 120, "rhf"),
        # a medium molecule in the throughput mode
        _case("block_mixed_w512_m76", "block", 512, 76, 10, 10, 400, "rhf", "mixed"),
        # production size: the throughput run of a large molecule on one GPU
        _case("block_mixed_w2048_m200", "block", 2048, 200, 32, 32, 1600, "rhf", "mixed"),
        # a user's own loop around the propagator, plain FP64: open-shell molecule
        _case("step_fp64_uhf_w640_m108", "step", 640, 108, 15, 15, 600, "uhf"),
        # the same, closed shell, larger batch
        _case("step_fp64_rhf_w1024_m160", "step", 1024, 160, 26, 26, 960, "rhf"),
        # mixed precision with unequal spin blocks and sizes that fill no tile
        _case("step_mixed_uhf_w700_m132", "step", 700, 132, 17, 14, 524, "uhf", "mixed"),
        # complex Cholesky vectors (spin-orbit or twisted boundary conditions)
        _case("step_complex_w256_m40", "step", 256, 40, 6, 5, 160, "complex"),
        # Green's functions and overlaps alone (estimators, back-propagation), odd sizes
        _case("greens_uhf_w777_m149", "greens", 777, 149, 23, 17, 0, "uhf"),
        # stabilisation of a large batch
        _case("reortho_rhf_w2048_m200", "reortho", 2048, 200, 32, 32, 0, "rhf"),
        # local energies in FP64, open shell
        _case("energy_fp64_uhf_w640_m108", "energy", 640, 108, 15, 15, 600, "uhf"),
        # local energies of the production size, mixed precision
        _case("energy_mixed_rhf_w2048_m200", "energy", 2048, 200, 32, 32, 1600, "rhf", "mixed"),
        # training or response through the local energy: forward and backward
        _case("gradient_uhf_w512_m76", "gradient", 512, 76, 10, 10, 400, "uhf"),
    ]


# real operations a drawn case may ask for, by kind and precision (a listed case's, or less)
_MOST = {("block", "fp64"): 4e11, ("block", "mixed"): 6e12, ("step", "fp64"): 1.6e11, ("step", "mixed"): 6e11,
         ("greens", "fp64"): 3e10, ("reortho", "fp64"): 3e10, ("energy", "fp64"): 4e11, ("energy", "mixed"): 2.8e12,
         ("gradient", "fp64"): 3e10}


def draw(rng):
    kind, precision, trial = rng.choice([
        ("block", "fp64", "rhf"), ("block", "mixed", "rhf"), ("block", "mixed", "uhf"), ("step", "fp64", "uhf"),
        ("step", "fp64", "rhf"), ("step", "mixed", "rhf"), ("step", "mixed", "uhf"), ("step", "fp64", "complex"),
        ("greens", "fp64", "uhf"), ("greens", "fp64", "rhf"), ("reortho", "fp64", "uhf"), ("reortho", "fp64", "rhf"),
        ("energy", "fp64", "uhf"), ("energy", "fp64", "rhf"), ("energy", "mixed", "rhf"), ("energy", "mixed", "uhf"),
        ("gradient", "fp64", "uhf")])
    mixed = precision == "mixed"
    M = int(round(math.exp(rng.uniform(math.log(20), math.log(80 if trial == "complex" else 200)))))
    X = int(M * rng.uniform(3.0, 8.0))
    if mixed:  # the mixed form takes multiples of 4
        M, X = (M + 3) // 4 * 4, (X + 3) // 4 * 4
    na = rng.randint(2, min(32, max(3, M // 5)))
    nb = na if trial == "rhf" else rng.randint(max(1, na - 6), na)
    W = int(round(math.exp(rng.uniform(math.log(8), math.log(2048)))))
    case = _case("", kind, W, M, na, nb, 0 if kind in ("greens", "reortho") else X, trial, precision)
    del case["name"]
    f = work(case)["flops"]
    if f > _MOST[kind, precision]:
        case["W"] = max(4, int(W * _MOST[kind, precision] / f))
    return case


def _flops(case):
    """(step, Green's function, reortho, energy) operations of the whole batch."""
    W, M, X = case["W"], case["M"], case["X"]
    spins = [case["na"]] if case["trial"] == "rhf" else [case["na"], case["nb"]]
    cplx = case["trial"] == "complex"
    fields = 2 * X if cplx else X
    green = sum(12 * M * n * n + 8 * n ** 3 for n in spins)
    reortho = sum(12 * M * n * n + 4 * n ** 3 for n in spins)
    bias = sum((8 if cplx else 4) * fields * n * M for n in spins)
    orbitals = sum((16 if cplx else 8) * M * M * n + 48 * M * M * n for n in spins)
    vhs = 8 * M * M * fields if cplx else 4 * (M * (M + 1) // 2) * X
    energy = sum(4 * X * n * n * M + 8 * X * n * n + 4 * X * n * M for n in spins)
    return W * (green + bias + orbitals + vhs), W * green, W * reortho, W * energy


def work(case):
    W, M, X = case["W"], case["M"], case["X"]
    spins = [case["na"]] if case["trial"] == "rhf" else [case["na"], case["nb"]]
    step, green, reortho, energy = _flops(case)
    phi = 16.0 * W * M * sum(spins)  # orbitals, or half-rotated Green's functions, of the batch
    half = 8.0 * X * M * sum(spins)  # half-rotated Cholesky vectors
    chol = 8.0 * X * (M * (M + 1) // 2)
    kind = case["kind"]
    if kind == "greens":
        return {"bytes": 2 * phi, "flops": green}
    if kind == "reortho":
        return {"bytes": 2 * phi, "flops": reortho}
    if kind == "energy":
        return {"bytes": phi + half + 48.0 * W, "flops": energy}
    if kind == "gradient":
        return {"bytes": 2 * phi + half + 16.0 * W, "flops": 3 * energy}
    if kind == "step":
        scale = 4 if case["trial"] == "complex" else 1
        return {"bytes": 2 * phi + scale * (half + chol) + 8.0 * W * X, "flops": step}
    return {"bytes": STEPS * (2 * phi + half + chol), "flops": STEPS * step + (STEPS // EVERY) * reortho + energy}


# ---------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float64)


def _system(case, seed):
    """h1 (M, M), Cholesky vectors (X, M, M) on the GPU and the trial orbitals of both spins.

    h1: diagonal linspace(-2, 1) plus N(0, 0.05) symmetric off-diagonals; vectors symmetric N(0, 1)
    with an exponential decay, scaled so that the auxiliary-field operator keeps a norm near 0.24;
    orbitals: the lowest eigenvectors of h1 plus the Hartree term, rotated per spin for "uhf"."""
    gen = _generator(seed)
    M, X, na, nb = case["M"], case["X"], case["na"], case["nb"]
    off = torch.triu(0.05 * _normal(gen, M, M), 1)
    h1 = torch.diag(torch.linspace(-2.0, 1.0, M, device="cuda", dtype=torch.float64)) + off + off.T
    decay = max(X, 1) / 8.0
    amp = 0.1 * math.sqrt(30.0 * 26.0 / (decay * M))
    chol = None
    fock = h1
    if X:
        scale = amp * torch.exp(-torch.arange(X, device="cuda", dtype=torch.float64) / decay)
        chol = _normal(gen, X, M, M)
        chol = (torch.triu(chol) + torch.triu(chol, 1).transpose(1, 2)) * scale[:, None, None]
        c0 = torch.linalg.eigh(h1)[1][:, :na]
        fock = h1 + torch.einsum("gpq,g->pq", chol, torch.einsum("gpq,pq->g", chol, c0 @ c0.T))
        if case["trial"] == "complex":
            chol = torch.complex(chol, 0.3 * _normal(gen, X, M, M) * scale[:, None, None])
    orbitals = torch.linalg.eigh(fock)[1]
    if case["trial"] == "rhf":
        return h1, chol, orbitals[:, :na].contiguous(), orbitals[:, :nb].contiguous()
    rot = 0.05 * _normal(gen, 2, M, M)
    rot = torch.linalg.matrix_exp(rot - rot.transpose(1, 2))
    return h1, chol, (rot[0] @ orbitals[:, :na]).contiguous(), (rot[1] @ orbitals[:, :nb]).contiguous()


def _trial_energy(h1, chol, psia, psib):
    """Energy of the trial determinant (its real vectors'), the shift that a walk's weights run at."""
    L = chol.real if chol.is_complex() else chol
    e, coul, exch = 5.0, 0.0, 0.0
    for psi in (psia, psib):
        t = psi.T @ L @ psi
        e = e + (psi * (h1 @ psi)).sum()
        coul = coul + t.diagonal(dim1=1, dim2=2).sum(dim=1)
        exch = exch + (t * t.transpose(1, 2)).sum()
    return float(e + 0.5 * (coul * coul).sum() - 0.5 * exch)


def _orbitals(case, seed, psia, psib):
    """Walkers as a walk leaves them: complex and near the trial."""
    gen = _generator(seed + 77777)
    W, s = case["W"], 0.3 / math.sqrt(case["M"])
    out = []
    for psi in (psia, psib):
        out.append((psi + s * torch.complex(_normal(gen, W, *psi.shape), _normal(gen, W, *psi.shape))).contiguous())
        if case["trial"] == "rhf":
            return out[0], out[0]
    return out


def _fields(case, seed):
    X = case["X"] * (2 if case["trial"] == "complex" else 1)
    return np.random.default_rng(seed + 5).normal(size=(2, case["W"], X))


def _objects(case, seed):
    """Hamiltonian, trial and walkers as a user's program builds them."""
    from ipie_b200 import Generic, SingleDet, UHFWalkers

    h1, chol, psia, psib = _system(case, seed)
    M, X, na, nb = case["M"], case["X"], case["na"], case["nb"]
    psi = torch.cat([psia, psib], dim=1).cpu().numpy()
    ham = None
    if X:
        h = h1.cpu().numpy()
        ham = Generic(np.array([h, h]), chol.reshape(X, M * M).T.contiguous().cpu().numpy(), 5.0)
    trial = SingleDet(psi, (na, nb), M)
    if ham is not None:
        trial.half_rotate(ham)
    walkers = UHFWalkers(psi, na, nb, M, case["W"])
    walkers.phia, walkers.phib = _orbitals(case, seed, psia, psib)
    if case["trial"] == "rhf":
        walkers.enable_spin_alias()
    walkers.build(trial)
    shift = _trial_energy(h1, chol, psia, psib) if case["kind"] == "step" else 0.0
    return ham, trial, walkers, shift


def prepare(case, seed):
    kind = case["kind"]
    ham, trial, walkers, shift = _objects(case, seed)
    state = dict(kind=kind, precision=case["precision"], ham=ham, trial=trial, walkers=walkers, k=0)
    if kind == "block":
        from ipie_b200 import AFQMC

        af = AFQMC.build((case["na"], case["nb"]), ham, trial, walkers=walkers, num_walkers=case["W"], seed=seed,
                         num_steps_per_block=STEPS, num_blocks=10 ** 6, timestep=DT, stabilize_freq=EVERY,
                         pop_control_freq=EVERY, verbose=False, rng="device", precision=case["precision"], graph=True,
                         population="device")
        af.setup_run()
        state["af"] = af
    elif kind == "step":
        from ipie_b200 import PhaselessGeneric, PopController

        prop = PhaselessGeneric(DT, rng="host", precision=case["precision"])
        prop.build(ham, trial, walkers)
        prop.host_fields = itertools.cycle([torch.from_numpy(a).pin_memory() for a in _fields(case, seed)])
        state.update(prop=prop, eshift=shift, pop=PopController(case["W"], STEPS, device=True))
    elif kind == "gradient":
        state["ghalf"] = [g.clone().requires_grad_(True) for g in (walkers.Ghalfa, walkers.Ghalfb)]
        state["upstream"] = torch.rand(case["W"], generator=_generator(seed + 3), device="cuda", dtype=torch.float64)
    elif kind == "energy" and case["precision"] == "mixed":
        from ipie_b200.estimators import _mixed_energy_operands, exchange_reference

        # laid out once per trial, as the estimator keeps them
        _mixed_energy_operands(trial, ham)
        exchange_reference(trial, ham)
    return state


def _walker_arrays(w):
    out = {"phia": w.phia, "weight": w.weight, "ovlp": w.ovlp, "ehyb": w.hybrid_energy}
    if not w.spin_alias:
        out["phib"] = w.phib
    return out


def run(state):
    kind, walkers, trial = state["kind"], state["walkers"], state["trial"]
    if kind == "block":
        af = state["af"]
        for _ in range(STEPS):
            state["k"] += 1
            af.step(state["k"])
        out = _walker_arrays(af.walkers)
        row = af.block_data[-1]
        out["energies"] = [float(row[0]), float(row[5]), float(row[6]), float(row[7])]
        return out
    if kind == "step":
        state["k"] += 1
        if state["k"] % EVERY == 0:
            walkers.reortho()
        state["prop"].propagate_walkers(walkers, state["ham"], trial, state["eshift"])
        if state["k"] % EVERY == 0:
            state["pop"].pop_control(walkers)
        return _walker_arrays(walkers)
    if kind == "greens":
        ovlp = trial.calc_greens_function(walkers)
        out = {"ghalfa": walkers.Ghalfa, "ovlp": ovlp}
        if not walkers.spin_alias:
            out["ghalfb"] = walkers.Ghalfb
        return out
    if kind == "reortho":
        det = walkers.reortho()
        out = {"phia": walkers.phia, "detR": det, "ovlp": walkers.ovlp}
        if not walkers.spin_alias:
            out["phib"] = walkers.phib
        return out
    if kind == "energy":
        from ipie_b200.estimators import local_energy_batch, local_energy_mixed

        f = local_energy_mixed if state["precision"] == "mixed" else local_energy_batch
        return f(None, state["ham"], walkers, trial)
    from ipie_b200.adjoint import LocalEnergyGreens

    ga, gb = state["ghalf"]
    e = LocalEnergyGreens.apply(ga, gb, state["ham"], trial)
    loss = (state["upstream"] * e.real).sum()
    da, db = torch.autograd.grad(loss, (ga, gb))
    return {"energy": e.detach(), "ga": da.conj(), "gb": db.conj()}  # conj(): the stored values, without a copy


# About four times and more of what the package shows against 64 bits.  FP64: rounding through the
# inverses and sums; a step's hybrid energy is a logarithm divided by dt, which costs three digits.
# Mixed: three-pass binary16 products with FP32 accumulation (about 1e-6 in a step's overlaps, 1e-5
# after a block's ten), the energies expanded around the trial's FP64 values (6e-9).  ``max`` leaves
# room for single values far below the others.
def tolerance(case):
    walk = case["kind"] in ("block", "step")
    if case["precision"] == "mixed":
        if not walk:
            return {"rel": 5e-8, "max": 1e-5}
        return {"rel": 1e-5 if case["kind"] == "step" else 1e-4, "max": 2e-2}
    return {"rel": 2e-10, "max": 1e-6} if walk else {"rel": 1e-12, "max": 1e-9}


# ---------------------------------------------------------------- 64-bit answers in plain torch
class _Exact:
    """The walk in complex128 torch on the same inputs."""

    def __init__(self, case, seed):
        self.case = case
        self.h1, self.chol, *psi = _system(case, seed)
        self.W, self.M, self.X = case["W"], case["M"], case["X"]
        phi = _orbitals(case, seed, *psi)
        self.shift = _trial_energy(self.h1, self.chol, *psi) if case["kind"] == "step" else 0.0
        self.n = 1 if case["trial"] == "rhf" else 2  # spin blocks computed; one block counts twice
        self.twice = 2.0 if self.n == 1 else 1.0
        self.psi, self.phi = psi[: self.n], list(phi[: self.n])
        self.weight = torch.ones(self.W, device="cuda", dtype=torch.float64)
        self.ehyb = torch.zeros(self.W, device="cuda", dtype=torch.complex128)
        self.greens()

    def greens(self):
        self.ghalf, ovlp = [], 1.0
        for psi, phi in zip(self.psi, self.phi):
            o = phi.transpose(1, 2) @ psi.to(phi.dtype)
            self.ghalf.append(torch.linalg.solve(o, phi.transpose(1, 2)))
            ovlp = ovlp * torch.linalg.det(o)
        self.ovlp = ovlp ** 2 if self.n == 1 else ovlp

    def reortho(self):
        det = 1.0
        for s, phi in enumerate(self.phi):
            q, r = torch.linalg.qr(phi)
            d = torch.diagonal(r, dim1=1, dim2=2)
            q = q * (d / d.abs())[:, None, :]
            self.phi[s] = q
            det = det * d.abs().prod(dim=1)
        det = det ** 2 if self.n == 1 else det
        self.ovlp = self.ovlp / det
        return det

    def setup(self):
        """Mean-field shift, one-body propagator and half-rotated vectors."""
        M, X = self.M, self.X
        L = self.chol.reshape(X, M * M)
        rho = [p @ torch.linalg.solve(p.T @ p, p.T) for p in self.psi]
        g = (rho[0] + (rho[0] if self.n == 1 else rho[1])).reshape(-1)
        flat = self.chol.permute(1, 2, 0).reshape(M, M * X)
        v0 = 0.5 * (flat @ flat.conj().T)
        if self.case["trial"] == "complex":
            A = 0.5 * (self.chol + self.chol.transpose(1, 2).conj())
            B = 0.5j * (self.chol - self.chol.transpose(1, 2).conj())
            self.ops = torch.cat([A, B]).reshape(2 * X, M * M)
            self.mf = 1j * (self.ops @ g.to(self.ops.dtype))
            h = (self.h1 - v0.real).to(self.ops.dtype)
        else:
            self.ops = L
            self.mf = 1j * (L @ g).to(torch.complex128)
            h = (self.h1 - v0).to(torch.complex128)
        shift = 1j * (self.mf @ self.ops.to(torch.complex128)).reshape(M, M)
        self.exp1 = torch.linalg.matrix_exp(-0.5 * DT * (h - shift))
        self.rot = [torch.einsum("xmn,mi->xin", self.ops.reshape(-1, M, M), p.to(self.ops.dtype)).reshape(
            self.ops.shape[0], -1).to(torch.complex128) for p in self.psi]

    def propagate(self, xi, eshift):
        """One phaseless step with the fields xi (W, fields)."""
        W, M, sdt = self.W, self.M, math.sqrt(DT)
        vbias = self.twice * sum(g.reshape(W, -1) @ r.T for g, r in zip(self.ghalf, self.rot))
        xbar = -sdt * (1j * vbias - self.mf)
        a = xbar.abs()
        xbar = torch.where(a > 1.0, xbar / a, xbar)
        xs = xi - xbar
        cmf = -sdt * (xs @ self.mf)
        cfb = (xi * xbar - 0.5 * xbar * xbar).sum(dim=1)
        for w in range(0, W, 512):
            x = xs[w:w + 512]
            if self.ops.is_complex():
                v = 1j * sdt * (x @ self.ops)
            else:
                v = 1j * sdt * torch.complex(x.real.contiguous() @ self.ops, x.imag.contiguous() @ self.ops)
            v = v.reshape(-1, M, M)
            for s in range(self.n):
                phi = self.exp1 @ self.phi[s][w:w + 512]
                t = phi
                for k in range(1, 7):
                    t = v @ t / k
                    phi = phi + t
                self.phi[s][w:w + 512] = self.exp1 @ phi
        old = self.ovlp
        self.greens()
        eh = -(torch.log(self.ovlp / old) + cfb + cmf) / DT
        bound = math.sqrt(2.0 / DT)
        if abs(eshift) >= 1e-10:
            eh = torch.complex(eh.real.clamp(eshift - bound, eshift + bound), eh.imag)
        growth = torch.exp(-DT * (0.5 * (eh.real + self.ehyb.real) - eshift))
        self.weight = self.weight * growth * torch.cos(-DT * eh.imag - cfb.imag).clamp(min=0.0)
        self.ehyb = eh

    def energy(self):
        """(W, 3) [total, one-body + core, two-body]."""
        out = [self.energy_of([g[w:w + 16] for g in self.ghalf]) for w in range(0, self.W, 16)]
        return torch.cat(out)

    def energy_of(self, gs):
        n, M, X = gs[0].shape[0], self.M, self.X
        e1, coul, exch = 5.0, 0.0, 0.0
        for s, g in enumerate(gs):
            N = g.shape[1]
            rh = (self.psi[s].T @ self.h1).to(g.dtype)
            e1 = e1 + self.twice * (g * rh).sum(dim=(1, 2))
            r = self.rot[s][:X]
            coul = coul + self.twice * (g.reshape(n, -1) @ r.T)
            t = (r.reshape(X * N, M) @ g.reshape(n * N, M).T).reshape(X, N, n, N)
            exch = exch + self.twice * torch.einsum("xinj,xjni->n", t, t)
        e2 = 0.5 * (coul * coul).sum(dim=1) - 0.5 * exch
        return torch.stack([e1 + e2, e1 + 0 * e2, e2], dim=1)

    def arrays(self):
        out = {"phia": self.phi[0], "weight": self.weight, "ovlp": self.ovlp, "ehyb": self.ehyb}
        if self.n == 2:
            out["phib"] = self.phi[1]
        return out


def _philox_normals(count, seed, block):
    """The package's device draws: Philox4x32-10 (Salmon et al., SC'11) counters (pair, block), 53-bit
    uniforms in (0, 1], Box-Muller."""
    pairs = (count + 1) // 2
    lo32, m32 = np.uint64(32), np.uint64(0xFFFFFFFF)
    x = [np.arange(pairs, dtype=np.uint64) & m32, np.arange(pairs, dtype=np.uint64) >> lo32,
         np.full(pairs, block, dtype=np.uint64), np.zeros(pairs, dtype=np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = x[0] * np.uint64(0xD2511F53), x[2] * np.uint64(0xCD9E8D57)
        x = [(p1 >> lo32) ^ x[1] ^ np.uint64(k0), p1 & m32, (p0 >> lo32) ^ x[3] ^ np.uint64(k1), p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF

    def uniform(a, b):
        v = ((a >> np.uint64(5)) << np.uint64(26)) | (b >> np.uint64(6))
        return torch.from_numpy((v.astype(np.float64) + 1.0) / 9007199254740992.0).cuda()

    u1, u2 = uniform(x[0], x[1]), uniform(x[2], x[3])
    rad = torch.sqrt(-2.0 * torch.log(u1))
    return torch.stack([rad * torch.cos(2 * math.pi * u2), rad * torch.sin(2 * math.pi * u2)], dim=1).reshape(-1)[:count]


def exact(case, seed):
    kind = case["kind"]
    ex = _Exact(case, seed)
    if kind == "greens":
        out = {"ghalfa": ex.ghalf[0], "ovlp": ex.ovlp}
        if ex.n == 2:
            out["ghalfb"] = ex.ghalf[1]
        return out
    if kind == "reortho":
        out = {"detR": ex.reortho(), "phia": ex.phi[0], "ovlp": ex.ovlp}
        if ex.n == 2:
            out["phib"] = ex.phi[1]
        return out
    ex.setup()
    if kind == "energy":
        return ex.energy()
    if kind == "gradient":
        up = torch.rand(case["W"], generator=_generator(seed + 3), device="cuda", dtype=torch.float64)
        e, da, db = [], [], []
        for w in range(0, ex.W, 16):
            gs = [g[w:w + 16].clone().requires_grad_(True) for g in ex.ghalf]
            part = ex.energy_of(gs)[:, 0]
            a, b = torch.autograd.grad((up[w:w + 16] * part.real).sum(), gs)
            e.append(part.detach())
            da.append(a.conj().resolve_conj())
            db.append(b.conj().resolve_conj())
        return {"energy": torch.cat(e), "ga": torch.cat(da), "gb": torch.cat(db)}
    if kind == "step":
        ex.propagate(torch.from_numpy(_fields(case, seed)[0]).cuda(), ex.shift)
        return ex.arrays()
    # block: ten steps at the shift 0 of a first block, weights rescaled at population control
    ex.reortho()
    total = 0.0
    bound = 0.1 * case["W"]
    for k in range(1, STEPS + 1):
        if k % EVERY == 0:
            ex.reortho()
        ex.propagate(_philox_normals(ex.W * ex.X, seed, k - 1).reshape(ex.W, ex.X), 0.0)
        if k > 1:
            ex.weight = ex.weight.clamp(-bound, bound)
        if k % EVERY == 0:
            s = float(ex.weight.abs().sum())
            bound = 0.1 * s
            ex.weight = ex.weight * (case["W"] / s)
            if float(ex.weight.min()) < 0.1 or float(ex.weight.max()) > 4.0:
                return None  # walkers branched: the pairing draws are not restated here
        total = total + float(ex.weight.sum())
    e = ex.energy().real
    mean = [float((ex.weight * e[:, k]).sum() / ex.weight.sum()) for k in range(3)]
    out = ex.arrays()
    out["energies"] = [total / STEPS] + mean
    return out
