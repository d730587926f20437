"""Performance cases: the propagation work users of this framework run, through its public calls.

A case names a workload (one drop-in step, an ensemble job, a group of aggregates, a loss gradient)
with its sizes.  prepare() builds what a program holds before the call, run() is one pass, work() the
bytes and operations a pass cannot do without, exact() the same outputs from plain complex128 torch:
the noise is drawn by its definition (Philox4x32-10, Box-Muller), every step is a Taylor series of
exp(-i H dt / hbar).

Outputs of mixed-precision jobs come from complex64 states, so they are returned in single precision,
which is what they carry; FP64 jobs return doubles.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

import dynaquant_b200 as dq
from dynaquant_b200 import _lib, systems

# ---------------------------------------------------------------------------------------------
# the cases


def listed():
    return [
        # One drop-in step per call: a host program that keeps its own state and steps one
        # trajectory at a time, asynchronously.  The chain is the smallest workload in use: launches
        # and latency are all of it.
        dict(name="step-chain", kind="step", system="chain", a=1024, b=1, m=16, dt=1.0),
        # The same call on the 30,000-site tube, the largest one a single trajectory is stepped on.
        dict(name="step-tube", kind="step", system="tube", a=60, b=500, m=20, dt=0.5),
        # The allocation-free step for programs that own all device memory, on the 5,278 sites and
        # m = 12 of the reference's example input, with its unconjugated dot product.
        dict(name="static-tube", kind="static", system="tube", a=58, b=91, m=12, dt=1.0),
        # The per-trajectory run of the example input: ZZ noise of 253 oscillators, static disorder,
        # the reference's own conventions, a few trajectories one after another.
        dict(name="plain-zz", kind="plain", system="tube", a=58, b=91, m=12, dt=1.0, noise="zz", B=2, steps=8),
        # A small FP64 ensemble: 64 trajectories on the chain, populations every 10 steps.
        dict(name="ens-chain-fp64", kind="ensemble", system="chain", a=1024, b=1, m=16, dt=1.0, noise="ou", B=64,
             steps=100, pop_every=10, precision="fp64", tuned=False),
        # A run of 100 trajectories, a number users write down, on a tube of odd size, untuned.
        dict(name="ens-odd", kind="ensemble", system="tube", a=57, b=83, m=20, dt=0.5, noise="ou", B=100, steps=32,
             pop_every=8, precision="mixed", tuned=False),
        # The benchmark workload: 256 trajectories on the 30,000-site tube, with the tiling that the
        # autotuner stored for it.
        dict(name="ens-tube", kind="ensemble", system="tube", a=60, b=500, m=20, dt=0.5, noise="ou", B=256, steps=16,
             pop_every=8, precision="mixed", tuned=True),
        # ZZ noise on a mid-size tube, as an input file runs it (no tuning), with the spectrum.
        dict(name="ens-zz", kind="ensemble", system="tube", a=60, b=68, m=20, dt=0.5, noise="zz", B=64, steps=48,
             pop_every=16, precision="mixed", tuned=False),
        # Many trajectories and long-range couplings (78 per row), tuned: the largest job.
        dict(name="ens-wide", kind="ensemble", system="tube", a=120, b=250, m=24, dt=0.5, noise="ou", B=1024,
             steps=3, pop_every=1, precision="mixed", tuned=True),
        # Uneven aggregates stepped together, each trajectory with its own Krylov dimension.
        dict(name="group-uneven", kind="group", a=60, lengths="34,68,135,270", trajectories="240,120,64,32", m=32,
             m_min=8, dt=0.5, steps=24),
        # One evaluation of a spectrum-fitting loss with its gradient (site energies, two scales).
        dict(name="gradient", kind="gradient", system="lattice", a=64, b=64, m=16, dt=1.0, B=128, steps=100,
             every=50, precision="mixed"),
        # Taylor-Krylov propagation of an ensemble (FP64).
        dict(name="taylor", kind="taylor", system="lattice", a=48, b=48, m=12, p=4, dt=1.0, B=32, steps=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "static", "plain", "ensemble", "ensemble", "ensemble", "group", "gradient", "taylor"])
    if kind in ("step", "static", "plain"):
        if rng.random() < 0.4:
            shape = dict(system="chain", a=_log(rng, 600, 20000), b=1)
        else:
            shape = dict(system="tube", a=rng.randint(17, 61), b=_log(rng, 30, 400))
        c = dict(kind=kind, **shape, m=rng.randint(8, 24), dt=rng.choice([0.5, 1.0]))
        if kind == "static":
            # the call's fixed scratch holds (m + 3) vectors
            c["m"] = min(c["m"], (16 * 2 ** 20 - 80000) // (16 * c["a"] * c["b"]) - 3)
        if kind == "plain":
            c.update(noise=rng.choice(["zz", "ou", "gauss"]), B=rng.randint(1, 4), steps=rng.randint(2, 8))
        return c
    if kind == "ensemble":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        if rng.random() < 0.3:
            shape = dict(system="chain", a=_log(rng, 500, 20000), b=1)
        else:
            shape = dict(system="tube", a=rng.randint(20, 64), b=_log(rng, 30, 500))
        n = shape["a"] * shape["b"]
        B = 2 * _log(rng, 8, 160)
        if rng.random() < 0.5:
            B = max(16, B // 16 * 16)
        noise = rng.choice(["ou", "ou", "gauss", "zz"])
        budget = 60e6 if precision == "mixed" and noise != "zz" else 20e6
        return dict(kind=kind, **shape, m=rng.randint(10, 24), dt=rng.choice([0.5, 1.0]), noise=noise, B=B,
                    steps=max(2, min(60, int(budget / (n * B)))), pop_every=rng.choice([1, 2, 5]), precision=precision,
                    tuned=precision == "mixed" and B % 16 == 0 and rng.random() < 0.5)
    if kind == "group":
        k = rng.randint(2, 4)
        ls = [_log(rng, 25, 250) for _ in range(k)]
        bs = [max(8, 8 * round(900 / x)) for x in ls]
        return dict(kind=kind, a=rng.randint(30, 60), lengths=",".join(map(str, ls)),
                    trajectories=",".join(map(str, bs)), m=rng.randint(20, 32), m_min=rng.choice([6, 8, 10]), dt=0.5,
                    steps=rng.randint(8, 24))
    side = rng.randint(20, 60)
    if kind == "gradient":
        return dict(kind=kind, system="lattice", a=side, b=side, m=rng.randint(10, 20), dt=rng.choice([0.5, 1.0]),
                    B=8 * rng.randint(2, 16), steps=rng.randint(20, 90), every=rng.choice([0, 16, 25]),
                    precision=rng.choice(["mixed", "fp64"]))
    return dict(kind=kind, system="lattice", a=side, b=side, m=rng.randint(6, 16), p=rng.randint(3, 6), dt=1.0,
                B=rng.randint(3, 32), steps=rng.randint(4, 12))


# ---------------------------------------------------------------------------------------------
# inputs

SIGMA, TAU, STATIC = 250.0, 50.0, 150.0        # OU / Gaussian noise (cm^-1, fs), static disorder
FFT = 4096                                     # spectrum length of the loss and of the ZZ job
STORED = {25.0: (16, 2, 1, 3, 12, 1), 40.0: (16, 2, 1, 3, 12, 4)}   # tilings a program keeps, by coupling cutoff


@functools.lru_cache(maxsize=24)
def _tube(a, b, cutoff):
    return systems.tube(a, b, cutoff=cutoff)


def _system(case):
    if case.get("system") == "chain":
        return systems.chain(case["a"])
    if case.get("system") == "lattice":
        return systems.lattice2d(case["a"])
    return _tube(case["a"], case["b"], _cutoff(case))


def _cutoff(case):
    return 40.0 if case["a"] >= 100 else 25.0


def _zz_density():
    om = 8.1357 * np.arange(1, 254)
    return om, 60.0 * (om / 120.0) * np.exp(-om / 120.0), 8.1357, 77.0


def _packet(n, seed):
    """A normalised complex state in mid-propagation: a random phase and size at every site."""
    g = np.random.default_rng(seed)
    v = g.normal(size=n) + 1j * g.normal(size=n)
    return v / np.linalg.norm(v)


def _start_state(case, s):
    """Chains start on their middle site; tubes and lattices from a bright state."""
    if case.get("system") == "chain":
        psi0 = np.zeros(s.n, dtype=np.complex128)
        psi0[s.n // 2] = 1.0
        return psi0
    return s.bright_state((1.0, 0.0, 0.0) if case.get("system") == "lattice" else (0.0, 0.0, 1.0))


_NOISE = {"none": dq.NOISE_NONE, "gauss": dq.NOISE_GAUSS, "ou": dq.NOISE_OU, "zz": dq.NOISE_ZZ}


def _set_noise(p, case, noise):
    if noise == "zz":
        p.set_zz_spectral_density(*_zz_density())
    else:
        p.set_noise_params(np.full(p.n, SIGMA), np.full(p.n, TAU))


def _site_energies(n, seed):
    return np.random.default_rng(seed + 1).normal(0.0, 100.0, n)


def _target(case, seed):
    """A measured spectrum to fit: one damped line, its place and width from the seed."""
    g = np.random.default_rng(seed + 2)
    k = np.arange(case["steps"] + 1)
    c = np.exp(-k / g.uniform(15.0, 40.0) - 1j * k * g.uniform(0.05, 0.3))
    return np.fft.ifft(c, FFT).real * FFT / case["steps"]


def _aux_matrix(s, seed):
    """The Taylor-Krylov auxiliary matrix B: the couplings on a diagonal of its own."""
    val = s.val.copy()
    rows = np.repeat(np.arange(s.n), np.diff(s.rowptr))
    on = rows == s.col
    val[on] = np.random.default_rng(seed + 3).normal(0.0, 60.0, int(on.sum()))
    return s.rowptr, s.col, val


def prepare(case, seed):
    kind = case["kind"]
    if kind == "group":
        members = []
        for i, (length, B) in enumerate(_members(case)):
            s = _tube(case["a"], length, 25.0)
            p = dq.Propagator(s.n, m=case["m"], n_traj=B, dt=case["dt"], noise=dq.NOISE_OU, sigma_static=STATIC,
                              seed=seed + 1000 * i, precision=dq.PREC_MIXED, pop_every=case["steps"],
                              max_steps=case["steps"], m_min=case["m_min"], m_tol=1e-7)
            p.set_system(s)
            p.set_noise_params(np.full(s.n, SIGMA), np.full(s.n, TAU))
            p.set_initial_state(s.bright_state())
            members.append(p)
        return dict(case=case, members=members, group=dq.Group(members))
    s = _system(case)
    if kind == "static":
        rp, col, val, _ = s.off_diagonal()
        diag = np.random.default_rng(seed).normal(0.0, SIGMA, s.n)
        psi = _packet(s.n, seed + 7)
        st = dict(case=case, n=s.n, lib=_lib.load())
        for name, arr in dict(rowptr=rp, col=col, val=val, diag=diag, psi=psi).items():
            st[name] = torch.from_numpy(np.ascontiguousarray(arr)).cuda()
        st["out"] = torch.zeros_like(st["psi"])
        torch.cuda.synchronize()
        return st
    noise = case.get("noise", "gauss" if kind == "step" else "ou")
    plain = kind in ("step", "plain")
    reference = kind == "plain"        # input-file runs keep the reference's conventions
    p = dq.Propagator(s.n, m=case["m"], n_traj=case.get("B", 1), dt=case["dt"], noise=_NOISE[noise],
                      sigma_static=0.0 if kind == "gradient" else STATIC, seed=seed,
                      dot=dq.DOT_BILINEAR if reference else dq.DOT_HERMITIAN,
                      norm=dq.NORM_REAL_ONLY if reference else dq.NORM_COMPLEX,
                      precision=dq.PREC_MIXED if case.get("precision") == "mixed" else dq.PREC_FP64,
                      pop_every=case.get("pop_every", 1), max_steps=max(case.get("steps", 1), 1))
    p.set_system(s)
    _set_noise(p, case, noise)
    st = dict(case=case, p=p)
    if kind == "gradient":
        p.set_coupling_classes(s.cls_off, [1.0, 1.0])
        p.set_static_energies(_site_energies(s.n, seed))
    p.set_initial_state(_start_state(case, s))
    if kind == "taylor":
        p.set_taylor_krylov(case["p"], case["m"], *_aux_matrix(s, seed))
    if kind == "gradient":
        p.adjoint_setup(case["steps"], FFT, 1.0 / case["steps"], _target(case, seed), checkpoint_every=case["every"])
    if case.get("tuned"):
        p.set_tiling(*STORED[_cutoff(case)])
    if kind == "step":
        st["psi"] = torch.from_numpy(_packet(s.n, seed + 7)).cuda()
        st["out"] = torch.zeros_like(st["psi"])
        p.reset()
    torch.cuda.synchronize()
    return st


def _members(case):
    return list(zip(map(int, case["lengths"].split(",")), map(int, case["trajectories"].split(","))))


# ---------------------------------------------------------------------------------------------
# one pass

STEP = 3   # index of the single steps


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        state["p"].prop_step(0, STEP, state["psi"].data_ptr(), state["out"].data_ptr())
        return state["out"]
    if kind == "static":
        t = state
        err = C.create_string_buffer(200)
        rc = t["lib"].dq_krylov_step_static(
            t["n"], t["rowptr"].data_ptr(), t["col"].data_ptr(), t["val"].data_ptr(), t["diag"].data_ptr(),
            t["psi"].data_ptr(), t["out"].data_ptr(), case["m"], case["dt"], 0.0, dq.DOT_BILINEAR, dq.NORM_REAL_ONLY,
            torch.cuda.current_stream().cuda_stream, None, err, len(err))
        if rc:
            raise dq.DQError(rc, err.value.decode())
        return t["out"]
    if kind == "plain":
        p = state["p"]
        p.run_plain(case["steps"])
        return p.populations(), p.correlation()
    if kind == "group":
        for p in state["members"]:
            p.reset()
        state["group"].run(case["steps"])
        return [(p.populations().astype(np.float32), p.correlation().astype(np.complex64)) for p in state["members"]]
    p = state["p"]
    if kind == "gradient":
        loss = p.forward()
        out = [np.array(loss), *p.backward()]
    else:
        p.reset()
        p.run(case["steps"])
        out = [p.populations(), p.correlation()]
        if case.get("noise") == "zz":
            out.append(p.spectrum(FFT))
    if case.get("precision") == "mixed":
        out = [x.astype(np.complex64 if x.dtype.kind == "c" else np.float32) for x in out]
    return out


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without


def work(case):
    """Per step and trajectory: the state in and out, the noise state, the Krylov basis written once
    and read once by the combination (a single step: its inputs and outputs only), m products with
    the couplings and the recurrence's vector operations."""
    kind = case["kind"]
    parts = _members(case) if kind == "group" else [(None, case.get("B", 1))]
    bytes_, flops = 0.0, 0.0
    for length, B in parts:
        s = _tube(case["a"], length, 25.0) if kind == "group" else _system(case)
        n, nnz, m = s.n, s.nnz - s.n, case["m"]
        steps = case.get("steps", 1)
        c = 8 if case.get("precision") == "mixed" or kind == "group" else 16
        if kind == "group":
            m = case["m_min"] + 4          # about the dimension the tolerance asks for
        iters = m + (case["p"] if kind == "taylor" else 0)
        flop = iters * (4.0 * nnz + 20.0 * n) + 8.0 * m * n
        if kind in ("step", "static", "plain"):
            traffic = 2.0 * 16 * n + 24.0 * n + 12.0 * nnz
        else:
            traffic = 2.0 * c * n + 24.0 * n + 2.0 * c * m * n
        if kind == "gradient":
            # the sweep: the second Krylov basis, the kept one read again, 2 m^2 + m products a site
            flop = 2.0 * flop + 8.0 * (2 * m * m + m) * n
            traffic = 2.0 * traffic + 2.0 * c * m * n
        bytes_ += steps * B * traffic
        flops += steps * B * flop
        if case.get("noise") == "zz":
            flops += steps * B * n * 253 * 4.0
    return dict(bytes=bytes_, flops=flops)


# ---------------------------------------------------------------------------------------------
# the same outputs in 64 bits

HBAR = (1 / 100.) * 1e15 / (299792548. * 2 * math.pi)
_M32 = 0xFFFFFFFF
_OU, _GAUSS, _OU_INIT, _STATIC, _ZZ = 1, 2, 3, 4, 5


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _philox(site, step, pair, word, seed):
    """Philox4x32-10 of the counter (site, step, pair, word) under the 64-bit seed, as int64 tensors."""
    c = [site & _M32, step + 0 * site, pair + 0 * site, word + 0 * site]
    c = list(torch.broadcast_tensors(*[x.to(torch.int64) for x in c]))
    k0, k1 = seed & _M32, (seed >> 32) & _M32
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
        p0, p1 = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
        c = [((p1 >> 32) & _M32) ^ c[1] ^ k0, p1 & _M32, ((p0 >> 32) & _M32) ^ c[3] ^ k1, p0 & _M32]
    return c


def _bits53(hi, lo):
    return (((hi << 32) | lo) >> 11) & ((1 << 53) - 1)


def _normals(seed, purpose, step, sub, n, B):
    """The [n, B] standard normals of one purpose, step and substep."""
    site = torch.arange(n, device=_dev())[:, None]
    pair = torch.arange((B + 1) // 2, device=_dev())[None, :]
    c = _philox(site + 0 * pair, torch.tensor(step, device=_dev()), pair + 0 * site,
                torch.tensor((purpose << 24) | sub, device=_dev()), seed)
    u1 = (_bits53(c[1], c[0]) + 1).double() * 2.0 ** -53
    u2 = _bits53(c[3], c[2]).double() * 2.0 ** -53
    r = torch.sqrt(-2.0 * torch.log(u1))
    z = torch.stack([r * torch.cos(2 * math.pi * u2), r * torch.sin(2 * math.pi * u2)], dim=2)
    return z.reshape(n, -1)[:, :B]


class _Diagonal:
    """The [n, B] site energies of consecutive steps."""

    def __init__(self, noise, static, n, B, dt, seed, eps=None):
        self.noise, self.n, self.B, self.dt, self.seed = noise, n, B, dt, seed
        self.eps = static * _normals(seed, _STATIC, 0, 0, n, B) if eps is None else eps[:, None]
        if noise == "ou":
            self.off = SIGMA * _normals(seed, _OU_INIT, 0, 0, n, B)
        if noise == "zz":
            om, J, d_om, T = _zz_density()
            G = J / (1 - np.exp(-om / (0.695035 * T)))
            self.amp = torch.from_numpy(np.sqrt(2.0) * np.sqrt(G * d_om / math.pi)).to(_dev())
            self.om = torch.from_numpy(om / 5308.84).to(_dev())
            self.re = self.im = None

    def at(self, k):
        if self.noise == "gauss":
            return self.eps + SIGMA * _normals(self.seed, _GAUSS, k, 0, self.n, self.B)
        if self.noise == "zz":
            site = torch.arange(self.n, device=_dev())[:, None]
            pair = torch.arange((self.B + 1) // 2, device=_dev())[None, :]
            sum_ = torch.zeros(self.n, pair.shape[1], 2, dtype=torch.float64, device=_dev())
            for o in range(len(self.om)):
                c = _philox(site + 0 * pair, torch.tensor(o, device=_dev()), pair + 0 * site,
                            torch.tensor(_ZZ << 24, device=_dev()), self.seed)
                u = torch.stack([_bits53(c[1], c[0]), _bits53(c[3], c[2])], dim=2).double() * 2.0 ** -53
                u = u.float().double()     # phases are kept in single precision
                u = torch.where(u >= 1.0, torch.zeros_like(u), u)
                sum_ += self.amp[o] * torch.cos(self.om[o] * (k * self.dt) + 2 * math.pi * u)
            return self.eps + sum_.reshape(self.n, -1)[:, :self.B]
        # OU: one Euler-Maruyama update before every step
        self.off = (self.off - self.off / TAU * self.dt
                    + SIGMA * math.sqrt(2.0 / TAU) * _normals(self.seed, _OU, k, 0, self.n, self.B) * math.sqrt(self.dt))
        return self.eps + self.off


class _Couplings:
    """Off-diagonal products: the k-th neighbour of every row at once."""

    def __init__(self, rowptr, col, val, n):
        rp = np.asarray(rowptr, dtype=np.int64)
        rows = np.repeat(np.arange(n), np.diff(rp))
        off = rows != col
        rows, col, val = rows[off], np.asarray(col)[off], np.asarray(val)[off]
        slot = np.arange(len(rows)) - np.searchsorted(rows, rows)
        K = int(slot.max()) + 1
        cols, vals = np.tile(np.arange(n), (K, 1)), np.zeros((K, n))
        cols[slot, rows], vals[slot, rows] = col, val
        self.cols = torch.from_numpy(cols).to(_dev())
        self.vals = torch.from_numpy(vals).to(_dev())
        self.place = (slot, rows)

    def __call__(self, x, vals=None):
        vals = self.vals if vals is None else vals
        y = torch.zeros_like(x)
        for k in range(len(self.cols)):
            y = y + vals[k][:, None] * x[self.cols[k]]
        return y


def _exp_step(x, apply, dt, terms=24):
    """exp(-i H dt / hbar) x as a Taylor series."""
    t, y = x, x
    for k in range(1, terms + 1):
        t = apply(t) * (-1j * dt / HBAR / k)
        y = y + t
    return y


def _unit(x):
    return x / torch.sqrt((x.real ** 2 + x.imag ** 2).sum(dim=0, keepdim=True))


def _exact_run(case, s, psi0, seed, noise, B, steps, pop_every, step=None):
    hop = _Couplings(s.rowptr, s.col, s.val, s.n)
    diagonal = _Diagonal(noise, STATIC, s.n, B, case["dt"], seed)
    bra = torch.from_numpy(psi0).to(_dev())[:, None]
    psi = bra.repeat(1, B)
    pops, corr = [bra[:, 0].abs() ** 2], [(bra.conj() * bra).sum()]
    aux = _Couplings(*_aux_matrix(s, seed), s.n) if case["kind"] == "taylor" else None
    if aux is not None:
        rows = np.repeat(np.arange(s.n), np.diff(s.rowptr))
        aux_diag = torch.from_numpy(_aux_matrix(s, seed)[2][rows == s.col]).to(_dev())[:, None]
    for k in range(steps):
        d = diagonal.at(k)
        if aux is None:
            psi = _unit(_exp_step(psi, lambda x: d * x + hop(x), case["dt"]))
        else:
            # sum_{q < p} (tau A)^q / q! psi + sum_{q >= p} tau^q B^(q - p) A^p / q! psi
            t, y = psi, psi
            for q in range(1, 30):
                t = (d * t + hop(t) if q <= case["p"] else aux_diag * t + aux(t)) * (-1j * case["dt"] / HBAR / q)
                y = y + t
            psi = _unit(y)
        corr.append((bra.conj() * psi).sum() / B)
        if (k + 1) % pop_every == 0:
            pops.append((psi.real ** 2 + psi.imag ** 2).mean(dim=1))
    return torch.stack(pops).cpu().numpy(), torch.stack(corr).cpu().numpy()


def _spectrum(corr, length):
    return np.fft.ifft(corr, length) * length


def exact(case, seed):
    kind = case["kind"]
    if kind == "group":
        out = []
        for i, (length, B) in enumerate(_members(case)):
            s = _tube(case["a"], length, 25.0)
            out.append(_exact_run(case, s, s.bright_state(), seed + 1000 * i, "ou", B, case["steps"], case["steps"]))
        return out
    s = _system(case)
    if kind in ("step", "static"):
        hop = _Couplings(s.rowptr, s.col, s.val, s.n)
        if kind == "static":
            d = torch.from_numpy(np.random.default_rng(seed).normal(0.0, SIGMA, s.n)).to(_dev())[:, None]
        else:
            d = _Diagonal("gauss", STATIC, s.n, 1, case["dt"], seed).at(STEP)
        psi = torch.from_numpy(_packet(s.n, seed + 7)).to(_dev())[:, None]
        return _unit(_exp_step(psi, lambda x: d * x + hop(x), case["dt"]))[:, 0]
    if kind == "gradient":
        return _exact_gradient(case, s, seed)
    noise = case.get("noise", "ou")
    out = list(_exact_run(case, s, _start_state(case, s), seed, noise, case["B"], case["steps"],
                          case.get("pop_every", 1)))
    if kind == "ensemble" and noise == "zz":
        out.append(_spectrum(out[1], FFT))
    return tuple(out) if kind == "plain" else out


def _exact_gradient(case, s, seed):
    from torch.utils.checkpoint import checkpoint
    n, B, T, dt = s.n, case["B"], case["steps"], case["dt"]
    eps = torch.from_numpy(_site_energies(n, seed)).to(_dev()).requires_grad_()
    scales = torch.ones(2, dtype=torch.float64, device=_dev(), requires_grad=True)
    hop = _Couplings(s.rowptr, s.col, s.val, n)
    cls = torch.zeros(hop.vals.shape, dtype=torch.int64, device=_dev())
    cls[hop.place] = torch.from_numpy(s.cls_off.astype(np.int64)).to(_dev())
    diagonal = _Diagonal("ou", 0.0, n, B, dt, seed, eps=torch.zeros(n, dtype=torch.float64, device=_dev()))
    bra = torch.from_numpy(_start_state(case, s)).to(_dev())[:, None]
    psi = bra.repeat(1, B)
    corr = [(bra.conj() * bra).sum()]

    def step(x, d, e, sc):
        vals = hop.vals * sc[cls]
        return _exp_step(x, lambda v: (d + e[:, None]) * v + hop(v, vals), dt, terms=18)

    for k in range(T):
        psi = checkpoint(step, psi, diagonal.at(k), eps, scales, use_reentrant=False)
        corr.append((bra.conj() * psi).sum() / B)
    spec = torch.fft.ifft(torch.stack(corr), FFT) * FFT
    target = torch.from_numpy(_target(case, seed)).to(_dev())
    loss = ((spec.real / T - target) ** 2).sum()
    gs, gc = torch.autograd.grad(loss, [eps, scales])
    return [loss.detach().cpu().numpy(), gs.cpu().numpy(), gc.cpu().numpy()]
