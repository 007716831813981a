"""The workloads that the framework's speed is measured on, each a call or two of its public API.

A case is a dict of plain values. `path` names the call:

* "block":   sampler.propagate_phaseless, one sampling block (phaseless steps, QR, local
             energies, stochastic reconfiguration), restarted from a saved population
* "driver":  driver.run_blocks, one driver block with the framework's own random draws
* "jvp", "vjp": the block's forward- and reverse-mode derivative with respect to h1
* "pair":    corr_sample.cs_block_scan, one correlated block of two Hamiltonians
* "free":    sampler.propagate_free, one free-projection block
* "cpmc":    propagator_cpmc.propagate, one constrained-path step of the Hubbard model
* "measure": trial.calc_overlap, calc_force_bias and calc_energy on one population

`precision` is the framework's own switch: "fp64" (complex128 walkers) or "mixed"
(complex64 walkers on the tensor cores). The mixed path's results carry single precision, so
a program keeps them in single precision, and so does run().

Hamiltonians are random with the shapes of real ones (no integral files here): symmetric
Cholesky vectors of falling size, h1 a spread of levels with noise, the trial its lowest
eigenvectors. Walkers are the trial plus complex noise, orthonormalised, as they are right
after a measurement.
"""

import math

import numpy as np
import torch

from cs_afqmc_gb300 import corr_sample, driver, hamiltonian, propagation, sampling, wavefunctions

F64, C128 = torch.float64, torch.complex128


def _case(name, path, precision, trial, norb, n_up, n_dn, nchol, nw, steps, lx=0, ly=0, restricted=True):
    return dict(name=name, path=path, precision=precision, trial=trial, norb=norb, n_up=n_up, n_dn=n_dn,
                nchol=nchol, nw=nw, steps=steps, lx=lx, ly=ly, restricted=restricted)


def listed():
    return [
        # the smallest calculation of the repository's workloads (50 walkers, 20 orbitals), as
        # its driver runs it: latency and launches
        _case("driver_fp64_norb20", "driver", "fp64", "rhf", 20, 5, 5, 100, 50, 5),
        # a small job of the serving stream: odd sizes, 64 walkers
        _case("block_mixed_norb53", "block", "mixed", "rhf", 53, 8, 8, 265, 64, 10),
        # the benchmark's molecule, five steps and a measurement
        _case("block_mixed_norb120", "block", "mixed", "rhf", 120, 20, 20, 600, 1024, 5),
        # the same molecule in the default precision, a quarter of the walkers
        _case("block_fp64_norb120", "block", "fp64", "rhf", 120, 20, 20, 600, 256, 5),
        # the 8 x 8 Hubbard lattice of the benchmark (diagonal Cholesky vectors)
        _case("block_mixed_hubbard8x8", "block", "mixed", "rhf", 64, 28, 28, 64, 2048, 5, 8, 8),
        # the upper end of the serving stream (norb up to 200, nocc = norb // 6)
        _case("block_mixed_norb198", "block", "mixed", "rhf", 198, 33, 33, 990, 256, 5),
        # the differentiation workload (UHF, 512 walkers): d energy / d lambda, and the 1-RDM
        _case("jvp_fp64_norb60", "jvp", "fp64", "uhf", 60, 10, 8, 300, 512, 3, restricted=False),
        _case("vjp_fp64_norb60", "vjp", "fp64", "uhf", 60, 10, 8, 300, 512, 3, restricted=False),
        # correlated sampling of h1 and h1 + lambda D on shared fields
        _case("pair_mixed_norb60", "pair", "mixed", "uhf", 60, 10, 8, 300, 512, 5, restricted=False),
        # free projection of a medium system
        _case("free_fp64_norb40", "free", "fp64", "uhf", 40, 7, 6, 200, 200, 5, restricted=False),
        # constrained path on the 8 x 8 lattice
        _case("cpmc_fp64_hubbard8x8", "cpmc", "fp64", "uhf", 64, 28, 28, 64, 512, 1, 8, 8, restricted=False),
        # measurements of a saved population, RHF trial on two-slab walkers
        _case("measure_fp64_norb80", "measure", "fp64", "rhf", 80, 13, 13, 400, 256, 1, restricted=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path, precision, trial = rng.choice([
        ("block", "mixed", "rhf"), ("block", "mixed", "rhf"), ("block", "mixed", "uhf"), ("block", "mixed", "hubbard"),
        ("block", "fp64", "rhf"), ("block", "fp64", "uhf"), ("driver", "fp64", "rhf"), ("driver", "mixed", "rhf"),
        ("jvp", "fp64", "uhf"), ("vjp", "fp64", "uhf"), ("jvp", "fp64", "rhf"), ("vjp", "fp64", "rhf"),
        ("pair", "mixed", "uhf"), ("pair", "fp64", "rhf"), ("free", "fp64", "uhf"), ("cpmc", "fp64", "uhf"),
        ("measure", "fp64", "rhf"), ("measure", "mixed", "uhf")])
    if trial == "hubbard" or path == "cpmc":
        lx, ly = rng.choice([(4, 4), (6, 4), (6, 6), (8, 6), (8, 8)])
        n = lx * ly
        nocc = rng.randint(n // 4, (7 * n) // 16)
        nw = _log_int(rng, 50, 2048 if path == "block" else 512)
        if path == "cpmc":
            return _case("", path, precision, "uhf", n, nocc, max(1, nocc - rng.randint(0, 2)), n, nw, 1, lx, ly, False)
        return _case("", path, precision, "rhf", n, nocc, nocc, n, nw, rng.randint(2, 6), lx, ly)
    top = {"block": 200 if precision == "mixed" else 120, "driver": 60}.get(path, 60 if path != "measure" else 100)
    norb = _log_int(rng, 16, top)
    n_up = max(2, norb // 6 + rng.randint(-1, 1))
    n_dn = n_up if trial == "rhf" else max(1, n_up - rng.randint(0, 2))
    nchol = max(8, int(norb * rng.uniform(3.0, 5.0)))
    most = 256 if norb > 128 else 1024 if precision == "mixed" else 256 if path == "block" else 300
    nw = _log_int(rng, 30, most)
    restricted = trial == "rhf" and (path != "measure") and rng.random() < 0.7
    steps = rng.randint(2, 5) if path not in ("jvp", "vjp") else rng.randint(1, 3)
    return _case("", path, precision, trial, norb, n_up, n_dn, nchol, nw, steps, 0, 0, restricted)


# ----------------------------------------------------------------------------- inputs

def _symmetric(x):
    u = torch.triu(x)
    return u + torch.triu(x, 1).transpose(-1, -2)


def _inputs(case, seed):
    """What a calculation starts from, as plain torch tensors on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 17)

    def randn(*shape):
        return torch.randn(shape, dtype=F64, device="cuda", generator=g)

    n, nw, nchol = case["norb"], case["nw"], case["nchol"]
    nelec = (case["n_up"], case["n_dn"])
    d = {"nelec": nelec, "dt": 0.005, "u": 4.0}
    if case["lx"]:
        lx, ly = case["lx"], case["ly"]
        h = np.zeros((n, n))
        for x in range(lx):
            for y in range(ly):
                for dx, dy in ((1, 0), (0, 1)):
                    j = ((x + dx) % lx) * ly + (y + dy) % ly
                    h[x * ly + y, j] -= 1.0
                    h[j, x * ly + y] -= 1.0
        h1 = torch.as_tensor(h, device="cuda")
        chol = torch.zeros((n, n, n), dtype=F64, device="cuda")
        i = torch.arange(n, device="cuda")
        chol[i, i, i] = math.sqrt(d["u"])
        levels = h1 + torch.diag(1e-3 * torch.linspace(-1.0, 1.0, n, dtype=F64, device="cuda"))
        d["dt"] = 0.01
        noise = 0.02
    else:
        size = torch.exp(-12.0 * torch.arange(nchol, dtype=F64, device="cuda") / nchol)
        size = size * torch.sqrt(12.5 / torch.sum(size * size)) * 0.5 / math.sqrt(n)
        chol = _symmetric(randn(nchol, n, n)) * size[:, None, None]
        h1 = 0.1 * _symmetric(randn(n, n)) + torch.diag(torch.linspace(-2.0, 2.0, n, dtype=F64, device="cuda"))
        levels = h1
        noise = 0.03
    # the trial: on the host, where eigenvectors of equal input come out equal
    v = np.linalg.eigh(levels.cpu().numpy())[1]
    if case["trial"] == "rhf":
        mo = [np.ascontiguousarray(v[:, :nelec[0]])] * 2
    else:
        r = np.random.default_rng(seed)
        mo = []
        for s in range(2):
            a = r.standard_normal((n, n)) * (0.05 if not case["lx"] else 0.01)
            q = np.linalg.qr(np.eye(n) + (a - a.T) / 2)[0]
            mo.append(np.ascontiguousarray((v @ q)[:, :nelec[s]]))
    d["mo"] = [torch.as_tensor(m, device="cuda") for m in mo]
    d["h1"], d["chol"] = torch.stack([h1, h1]), chol
    walkers = []
    for s in range(1 if case["restricted"] else 2):
        re = d["mo"][s][None] + noise * randn(nw, n, nelec[s])
        if case["path"] == "cpmc":
            w = re
        else:
            w = torch.complex(re, noise * randn(nw, n, nelec[s]))
            w = _householder_q(w)[0]
        if case["precision"] == "mixed":
            w = w.to(torch.complex64)
        walkers.append(w.contiguous())
    d["walkers"] = walkers
    d["weights"] = 0.6 + 0.8 * torch.rand((nw,), dtype=F64, device="cuda", generator=g)
    d["fields"] = randn(1, 1, case["steps"], nw, nchol) if case["path"] != "driver" else None
    d["zetas"] = torch.rand((1,), dtype=F64, device="cuda", generator=g)
    d["op"] = _symmetric(randn(n, n)) / n
    return d


def prepare(case, seed):
    d = _inputs(case, seed)
    n, nw, nelec = case["norb"], case["nw"], d["nelec"]
    restricted, path = case["restricted"], case["path"]
    uhf = case["trial"] == "uhf"
    ham = hamiltonian.hamiltonian(n)
    rdm1 = torch.stack([m @ m.T for m in d["mo"]])
    wave = {"mo_coeff": d["mo"] if uhf else d["mo"][0], "rdm1": rdm1}
    if path == "cpmc":
        trial = wavefunctions.uhf_cpmc(n, nelec)
        prop = propagation.propagator_cpmc(dt=d["dt"], n_walkers=nw)
    else:
        trial = (wavefunctions.uhf if uhf else wavefunctions.rhf)(n, nelec)
        kind = propagation.propagator_restricted if restricted else propagation.propagator_unrestricted
        prop = kind(dt=d["dt"], n_walkers=nw, precision=case["precision"])
    samp = sampling.sampler(n_prop_steps=case["steps"], n_ene_blocks=1, n_sr_blocks=1, n_blocks=1)
    init = [w.to(C128) for w in d["walkers"]] if path == "cpmc" else d["walkers"]
    init = init[0] if restricted else init
    s = {"case": case, "d": d, "ham": ham, "trial": trial, "prop": prop, "samp": samp, "wave": wave, "systems": []}
    for k in range(2 if path == "pair" else 1):
        h1 = d["h1"] + (0.0 if k == 0 else 0.05) * d["op"]
        hd = {"h0": 0.0, "h1": h1, "chol": d["chol"].reshape(case["nchol"], n * n), "ene0": 0.0, "u": d["u"]}
        hd = ham.build_measurement_intermediates(hd, trial, wave)
        hd = ham.build_propagation_intermediates(hd, prop, trial, wave)
        own = [w.clone() for w in init] if isinstance(init, list) else init.clone()
        pd = prop.init_prop_data(trial, wave, hd, init_walkers=own)
        pd["weights"].copy_(d["weights"])
        pd["key"] = propagation.RngKey(int(seed) + 5)
        s["systems"].append((hd, pd, _saved(pd)))
    return s


_SAVED = ("walkers", "weights", "overlaps", "_scalars", "norms", "normed_overlaps", "greens")


def _saved(pd):
    """A copy of the population, as a program keeps to restart from."""
    return {k: [x.clone() for x in pd[k]] if isinstance(pd[k], list) else pd[k].clone() for k in _SAVED if k in pd}


def _restart(pd, saved):
    for k in ("walkers", "weights", "_scalars"):
        for dst, src in zip(pd[k], saved[k]) if isinstance(saved[k], list) else ((pd[k], saved[k]),):
            dst.copy_(src)


def _single(case, x):
    if case["precision"] != "mixed":
        return x
    return x.to(torch.complex64) if x.is_complex() else x.to(torch.float32)


def run(s):
    case, d, ham, trial, prop, samp, wave = (s[k] for k in ("case", "d", "ham", "trial", "prop", "samp", "wave"))
    hd, pd, saved = s["systems"][0]
    path = case["path"]
    one = lambda x: _single(case, x)  # noqa: E731
    if path == "measure":
        w = pd["walkers"]
        return {"overlaps": one(trial.calc_overlap(w, wave)), "force_bias": one(trial.calc_force_bias(w, hd, wave)),
                "energies": one(trial.calc_energy(w, hd, wave))}
    if path == "driver":  # goes on from the population as the last block left it
        be, bw, pd = driver.run_blocks(samp, ham, hd, prop, pd, trial, wave, 1)
        return {"energy": one(be), "weight": one(bw), "weights": one(pd["weights"]), "walkers": pd["walkers"]}
    _restart(pd, saved)
    if path == "block":
        e, pd = samp.propagate_phaseless(ham, hd, prop, pd, trial, wave, fields=d["fields"], zetas=d["zetas"])
        return {"energy": one(e), "block_weights": one(pd["block_weights"]), "weights": one(pd["weights"]),
                "overlaps": one(pd["overlaps"]), "walkers": pd["walkers"]}
    if path == "jvp":
        e, de, pd = samp.propagate_phaseless_ad_norot_jvp(ham, hd, d["op"], prop, pd, trial, wave,
                                                          fields=d["fields"], zetas=d["zetas"])
        return {"energy": e, "denergy": de, "weights": pd["weights"], "walkers": pd["walkers"]}
    if path == "vjp":
        e, rdm1, pd = samp.propagate_phaseless_ad_norot_vjp(ham, hd, prop, pd, trial, wave,
                                                            fields=d["fields"], zetas=d["zetas"])
        return {"energy": e, "rdm1": rdm1, "weights": pd["weights"], "walkers": pd["walkers"]}
    if path == "pair":
        hd2, pd2, saved2 = s["systems"][1]
        _restart(pd2, saved2)
        for p, q in ((pd, saved), (pd2, saved2)):  # the block's steps start from the overlaps
            p["overlaps"].copy_(q["overlaps"])
        sums = torch.empty(4, dtype=F64, device="cuda")
        corr_sample.cs_block_scan(pd, hd, prop, trial, wave, pd2, hd2, prop, trial, wave, samp,
                                  fields=d["fields"], sums=sums)
        return {"sums": one(sums), "weights": [one(pd["weights"]), one(pd2["weights"])],
                "walkers": [pd["walkers"], pd2["walkers"]]}
    if path == "free":
        for k in ("norms", "normed_overlaps"):
            pd[k] = saved[k].clone()
        pd, be, bw, _ = samp.propagate_free(ham, hd, prop, pd, trial, wave, fields=d["fields"][0])
        return {"energy": be, "weight": bw, "overlaps": pd["overlaps"], "norms": pd["norms"],
                "normed_overlaps": pd["normed_overlaps"], "walkers": pd["walkers"]}
    # cpmc: one step with Gaussians for the site fields
    pd["overlaps"].copy_(saved["overlaps"])
    pd["greens"].copy_(saved["greens"])
    pd = prop.propagate(trial, hd, pd, d["fields"][0, 0, 0], wave)
    return {"walkers": pd["walkers"], "weights": pd["weights"], "overlaps": pd["overlaps"], "greens": pd["greens"]}


# ----------------------------------------------------------------------------- 64-bit values

def _householder_q(a):
    """(Q, prod diag R) of the reduced QR with LAPACK's signs, [nw, n, k], differentiable."""
    n, k = a.shape[-2:]
    vs, taus, rprod = [], [], 1.0
    for j in range(k):
        x = a[..., j:, j]
        norm = torch.sqrt(torch.sum((x * x.conj()).real, -1))
        alpha = x[..., 0]
        beta = torch.where(alpha.real >= 0, -norm, norm).to(a.dtype)
        tau = (beta - alpha) / beta
        v = torch.cat([torch.ones_like(alpha)[..., None], x[..., 1:] / (alpha - beta)[..., None]], -1)
        v = torch.nn.functional.pad(v, (j, 0))
        a = a - tau.conj()[..., None, None] * v[..., :, None] * torch.matmul(v.conj()[..., None, :], a)
        vs.append(v)
        taus.append(tau)
        rprod = rprod * beta
    q = torch.eye(n, k, dtype=a.dtype, device=a.device).expand(a.shape)
    for v, tau in zip(reversed(vs), reversed(taus)):
        q = q - tau[..., None, None] * v[..., :, None] * torch.matmul(v.conj()[..., None, :], q)
    return q, rprod


class _Exact:
    """The phaseless path in plain 64-bit torch, differentiable in h1."""

    def __init__(self, case, d, h1, walkers=None):
        self.case, self.d, self.dt = case, d, d["dt"]
        n = case["norb"]
        mo, chol = d["mo"], d["chol"]
        self.mo, self.chol, self.uhf, self.two = mo, chol, case["trial"] == "uhf", not case["restricted"]
        h1 = torch.stack([(h1[s] + h1[s].T) / 2 for s in range(2)])
        rho = sum(m @ m.T for m in mo)
        self.mf = torch.complex(torch.zeros_like(chol[:, 0, 0]), torch.einsum("gij,ij->g", chol, rho))
        v0 = 0.5 * torch.einsum("gik,gjk->ij", chol, chol)
        v1 = -torch.einsum("g,gij->ij", self.mf.imag, chol)
        if self.two:
            self.expm = [torch.matrix_exp(-self.dt * (h1[s] - v0 - v1) / 2).to(C128) for s in range(2)]
        else:
            self.expm = [torch.matrix_exp(-self.dt * ((h1[0] + h1[1]) / 2 - v0 - v1) / 2).to(C128)]
        self.h0_prop = -torch.sum(self.mf * self.mf).real / 2
        spin_h1 = [h1[s] if self.uhf else (h1[0] + h1[1]) / 2 for s in range(2)]
        self.rot_h1 = [(mo[s].T @ spin_h1[s]).to(C128) for s in range(2)]
        self.rc = [torch.einsum("pi,gpj->gij", mo[s], chol) for s in range(2 if self.uhf else 1)]
        self.w = [w.to(C128) for w in (d["walkers"] if walkers is None else walkers)]
        self.weights = d["weights"]
        self.ovl = self.overlap()
        self.e_est = self.energies().real.sum().detach() / case["nw"]
        self.pcs = self.e_est

    def overlap(self):
        o = 1.0
        for s, w in enumerate(self.w):
            o = o * torch.linalg.det(self.mo[s].T.to(C128) @ w)
        return o if self.two else o * o

    def green(self):
        g = [(w @ torch.linalg.inv(self.mo[s].T.to(C128) @ w)).transpose(1, 2) for s, w in enumerate(self.w)]
        return g if self.uhf or len(g) == 1 else [g[0] + g[1]]

    @staticmethod
    def _mm(a, b):
        """complex [nw, k] times real [k, m]"""
        return torch.complex(a.real @ b, a.imag @ b)

    def force_bias(self):
        fb = sum(self._mm(g.reshape(g.shape[0], -1), rc.reshape(rc.shape[0], -1).T) for g, rc in zip(self.green(), self.rc))
        return fb if self.two else 2 * fb

    def energies(self):
        out, gr = [], self.green()
        nw, nchol = self.case["nw"], self.case["nchol"]
        occ = max(self.d["nelec"])
        step = max(1, int(2e8 / (nchol * occ * occ)))
        for a in range(0, nw, step):
            g = [x[a:a + step] for x in gr]
            e1 = sum(torch.einsum("wip,ip->w", x, r) for x, r in zip(g, self.rot_h1))
            exc, coul = 0.0, []
            for x, rc in zip(g, self.rc):
                m, o, n = x.shape
                f = self._mm(x.reshape(m * o, n), rc.reshape(-1, n).T).reshape(m, o, nchol, o)
                exc = exc + torch.einsum("wkgi,wigk->w", f, f)
                coul.append(torch.einsum("wigi->wg", f))
            if not self.two:
                e = 2 * e1 + 2 * torch.sum(coul[0] ** 2, 1) - exc
            elif not self.uhf:
                e = e1 + torch.sum(coul[0] ** 2, 1) - exc
            else:
                e = e1 + 0.5 * (torch.sum((coul[0] + coul[1]) ** 2, 1) - exc)
            out.append(e)
        return torch.cat(out)

    def apply(self, xt):
        n = self.case["norb"]
        v = 1j * math.sqrt(self.dt) * self._mm(xt, self.chol.reshape(-1, n * n)).reshape(-1, n, n)
        out = []
        for e, w in zip(self.expm, self.w):
            t = e @ w
            acc = t
            for m in range(1, 6):
                t = v @ t / m
                acc = acc + t
            out.append(e @ acc)
        self.w = out

    def step(self, x):
        sq = math.sqrt(self.dt)
        s = -sq * (1j * self.force_bias() - self.mf)
        xt = x - s
        shift = torch.sum(xt * self.mf, 1)
        fbt = torch.sum(x * s - s * s / 2, 1)
        self.apply(xt)
        new = self.overlap()
        arg = (-sq * shift + fbt).real + self.dt * (self.pcs + self.h0_prop)
        phase = torch.polar(torch.ones_like(arg), (-sq * shift).imag)
        imp = torch.exp(arg) * (phase * new / self.ovl).real
        imp = torch.where(torch.isnan(imp) | (imp < 1e-3) | (imp > 100), torch.zeros_like(imp), imp)
        w = imp * self.weights
        self.weights = torch.where(w > 100, torch.zeros_like(w), w)
        self.pcs = self.e_est - 0.1 * torch.log(torch.sum(self.weights) / self.case["nw"]) / self.dt
        self.ovl = new

    def block(self, fields):
        for x in fields:
            self.step(x)
        self.w = [_householder_q(w)[0] for w in self.w]
        self.ovl = self.overlap()
        e = self.energies().real
        self.local = torch.where(torch.abs(e - self.e_est) > math.sqrt(2 / self.dt), self.e_est, e)
        self.block_weight = torch.sum(self.weights)
        return torch.sum(self.local * self.weights) / self.block_weight

    def reconfigure(self, zeta):
        nw = self.case["nw"]
        cum = torch.cumsum(self.weights.detach().abs(), 0)
        z = cum[-1] * (torch.arange(nw, dtype=F64, device="cuda") + zeta) / nw
        idx = torch.searchsorted(cum, z).clamp(max=nw - 1)
        self.weights = (torch.sum(self.weights) / nw).expand(nw)
        self.w = [w[idx] for w in self.w]
        self.ovl = self.overlap()

    def walkers(self):
        w = [x.detach() for x in self.w]
        return w if self.two else w[0]


def _exact_free(case, d):
    x = _Exact(case, d, d["h1"])
    nw, nel, sq = case["nw"], d["nelec"], math.sqrt(d["dt"])
    norms = torch.ones(nw, dtype=C128, device="cuda")
    for f in d["fields"][0, 0]:
        s = f.to(C128) @ x.mf
        x.apply(f.to(C128))
        qs = []
        for k, w in enumerate(x.w):
            c = torch.exp(-sq * s / (2 * nel[k]) + d["dt"] * x.h0_prop / (2 * nel[k]))
            q, r = _householder_q(c[:, None, None] * w)
            qs.append(q)
            norms = norms * r
        x.w = qs
    o = x.overlap() * norms
    e = x.energies()
    walkers = x.walkers()
    x.w = [_householder_q(w)[0] for w in x.w]
    return {"energy": (torch.sum(e * o) / torch.sum(o)).reshape(1), "weight": torch.sum(o).reshape(1), "overlaps": o,
            "norms": norms, "normed_overlaps": x.overlap(), "walkers": walkers}


def _exact_cpmc(case, d):
    x = _Exact(case, d, d["h1"], [w.to(C128) for w in d["walkers"]])
    pcs, dt, n = x.e_est, d["dt"], case["norb"]
    mo, expm = d["mo"], [e.real for e in x.expm]
    w, weights, ovl = [a.clone() for a in d["walkers"]], d["weights"].clone(), x.ovl.real
    gamma, c = math.acosh(math.exp(dt * d["u"] / 2)), math.exp(-dt * d["u"] / 2)
    hs = torch.tensor([[c * math.exp(gamma), c * math.exp(-gamma)], [c * math.exp(-gamma), c * math.exp(gamma)]],
                      dtype=F64, device="cuda")

    def one_body():
        nonlocal weights, ovl
        new, g = 1.0, []
        for s in range(2):
            w[s] = expm[s] @ w[s]
            m = mo[s].T @ w[s]
            new = new * torch.linalg.det(m)
            g.append((w[s] @ torch.linalg.inv(m) @ mo[s].T).transpose(1, 2))
        weights = weights * new / ovl
        weights = torch.where(weights < 1e-8, torch.zeros_like(weights), weights)
        ovl = new
        return g

    g = one_body()
    uni = (torch.erf(d["fields"][0, 0, 0] / math.sqrt(2.0)) + 1) / 2
    eye = torch.eye(n, dtype=F64, device="cuda")
    for i in range(n):
        diag = [g[s][:, i, i] for s in range(2)]
        r = torch.stack([(1 + (hs[f, 0] - 1) * diag[0]) * (1 + (hs[f, 1] - 1) * diag[1]) for f in range(2)])
        r = torch.where(r < 1e-8, torch.zeros_like(r), r)
        norm = (r[0] + r[1]) / 2
        f = torch.where(uni[:, i] < r[0] / 2 / norm, 0, 1)
        ratio = torch.where(f == 0, r[0], r[1])
        weights, ovl = weights * norm, ovl * ratio
        u = hs[f] - 1
        for s in range(2):
            w[s][:, i] *= hs[f, s][:, None]
        col = [g[s][:, :, i] for s in range(2)]
        row = [g[s][:, i, :] - eye[i] for s in range(2)]
        g = [g[s] + (u[:, s] / ratio)[:, None, None] * col[s][:, :, None] *
             (-(u[:, 1 - s] * diag[1 - s] + 1)[:, None] * row[s])[:, None, :] for s in range(2)]
    g = one_body()
    weights = weights * math.exp(dt * float(pcs))
    weights = torch.where(weights > 100, torch.zeros_like(weights), weights)
    return {"walkers": w, "weights": weights, "overlaps": ovl, "greens": torch.stack(g, 1)}


def exact(case, seed):
    path = case["path"]
    if path == "driver":  # the fields are the framework's own draws
        return None
    d = _inputs(case, seed)
    if path == "measure":
        x = _Exact(case, d, d["h1"])
        return {"overlaps": x.ovl, "force_bias": x.force_bias(), "energies": x.energies()}
    if path == "free":
        return _exact_free(case, d)
    if path == "cpmc":
        return _exact_cpmc(case, d)
    fields = d["fields"][0, 0]
    if path == "pair":
        x = [_Exact(case, d, d["h1"] + a * d["op"]) for a in (0.0, 0.05)]
        for y in x:
            y.block(fields)
        z = [torch.abs(y.weights - y.weights.mean()) / y.weights.std(unbiased=False) for y in x]
        keep = torch.where(z[0] > z[1], z[0], z[1]) <= 5.0
        w = [torch.where(keep, y.weights, torch.zeros_like(y.weights)) for y in x]
        sums = torch.stack([v for y, u in zip(x, w) for v in (torch.sum(y.local * u), torch.sum(u))])
        return {"sums": sums, "weights": w, "walkers": [y.walkers() for y in x]}
    h1 = d["h1"].clone().requires_grad_(path in ("jvp", "vjp"))
    x = _Exact(case, d, h1)
    e = x.block(fields)
    bw = x.block_weight
    grad = torch.autograd.grad(e, h1)[0] if h1.requires_grad else None
    with torch.no_grad():
        x.reconfigure(d["zetas"][0])
    weights = x.weights.detach().clone()
    if path == "jvp":
        return {"energy": e.detach(), "denergy": torch.sum(grad * torch.stack([d["op"]] * 2)), "weights": weights,
                "walkers": x.walkers()}
    if path == "vjp":
        return {"energy": e.detach(), "rdm1": grad, "weights": weights, "walkers": x.walkers()}
    return {"energy": e, "block_weights": bw.reshape(1), "weights": weights, "overlaps": x.ovl, "walkers": x.walkers()}


# ----------------------------------------------------------------------------- work

def work(case):
    """Bytes and operations one pass cannot do without: the inputs (Cholesky vectors, fields,
    population) read once, the outputs written once; the dense contractions of each step and
    of the measurement."""
    n, g, nw, steps, path = case["norb"], case["nchol"], case["nw"], case["steps"], case["path"]
    occ = [case["n_up"]] if case["restricted"] else [case["n_up"], case["n_dn"]]
    pop = nw * n * sum(occ) * (8 if case["precision"] == "mixed" else 16)
    if path == "cpmc":
        flops = nw * sum(2 * 2 * n * n * o + 2 * (4 * n * o * o + 2 * n * n * o + 2 * o ** 3) + 3 * n ** 3 for o in occ)
        return {"bytes": pop + 8 * nw * n + 8 * 2 * nw * n * n, "flops": flops}
    spins = occ if case["trial"] == "uhf" else occ[:1]
    rows = g if not case["lx"] else 1  # on a lattice each vector has one entry
    green = sum(6 * n * o * o * 2 + 8 * o ** 3 for o in occ)
    fb = sum(4 * g * o * n for o in spins)
    energy = sum(4 * min(g * o * o * n, (o * n) ** 2) for o in spins) + fb
    step = fb + (4 * g * n * n if not case["lx"] else 4 * g) + sum(5 * 8 * n * n * o + 2 * 4 * n * n * o for o in occ) + green
    if case["lx"]:
        step -= sum(5 * 8 * n * n * o - 5 * 8 * n * o for o in occ)
    qr = sum(16 * n * o * o for o in occ)
    if path == "free":
        step = step - fb - green + 2 * qr
    block = steps * step + qr + energy + green
    ham = 8 * (rows * n * n if not case["lx"] else g) + 8 * g * n * sum(spins)
    if path == "measure":
        return {"bytes": ham - 8 * g * n * n + pop + 16 * nw * (g + 2), "flops": nw * (2 * green + fb + energy)}
    flops = nw * block * {"jvp": 2.5, "vjp": 3.0, "pair": 2.0}.get(path, 1.0)
    size = ham + 2 * pop + 8 * nw * g * steps
    return {"bytes": size + (ham + 2 * pop if path == "pair" else 0), "flops": flops}
