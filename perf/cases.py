"""The work this force field is used for, as measurable cases.

Every case goes through the public Python entry points (moldy_gb300.forcefield, .dynamics, .fitting) as a user's
program does.  The forms and sizes are those of the repository's workloads: argon without charges, rigid 4-site water,
MCY-potential water, rock salt, water over a framework, force-matching fits and dynamics, from some hundred sites to
131,072.

The FP64 form's results are handed on as float64.  The mixed form computes in FP32 (forces good to about 1e-7 to 1e-6 of
their size), and a program that selects it keeps its results in float32, which is what those cases return.
"""
import math

import numpy as np
import torch

from moldy_gb300 import system as S
from moldy_gb300.dynamics import MolecularDynamics, species_dynamics, thermal_state
from moldy_gb300.fitting import FitProblem, ForceMatchLoss, water_frames
from moldy_gb300.forcefield import ForceField


def listed():
    return [
        # The smallest call: one host-array force evaluation of a Lennard-Jones solid without charges (a thousand-step
        # run of 500 atoms makes one per step); launches and copies are all of it.
        {"name": "argon500_fp64", "kind": "forces", "system": "argon", "n": 5, "form": "fp64", "strict": True},
        # The small water box of the parity and drift runs, in the form that production uses and in the FP64 form.
        {"name": "water2048_mixed", "kind": "forces", "system": "water", "n": 8, "form": "mixed", "strict": False},
        {"name": "water2048_fp64", "kind": "forces", "system": "water", "n": 8, "form": "fp64", "strict": False},
        # Water over a charged framework (clay-like systems): an odd number of sites, framework exclusions in both parts.
        {"name": "waterwall1044_mixed", "kind": "forces", "system": "wall", "n": 7, "form": "mixed", "strict": False},
        # The two calls that the reference's own step makes, force_calc then ewald, adding into host arrays: MCY water of
        # an odd size with the strict cut-off.
        {"name": "mcy8788_strict_mixed", "kind": "calls", "system": "mcy", "n": 13, "form": "mixed", "strict": True},
        # An ionic crystal listed species by species (Buckingham + Ewald), every site charged, host arrays.
        {"name": "rocksalt32768_mixed", "kind": "forces", "system": "rocksalt", "n": 16, "form": "mixed", "strict": False},
        # The large water box with everything on the device, as a GPU-resident integrator calls it; both forms.
        {"name": "water131072_mixed", "kind": "device", "system": "water", "n": 32, "form": "mixed", "strict": False},
        {"name": "water131072_fp64", "kind": "device", "system": "water", "n": 32, "form": "fp64", "strict": False},
        # Force matching: loss and gradient (forward and backward through torch) over a batch of frames.
        {"name": "fit16384_mixed", "kind": "fit", "system": "water", "n": 16, "form": "mixed", "strict": False, "frames": 4},
        {"name": "fit2048_fp64", "kind": "fit", "system": "water", "n": 8, "form": "fp64", "strict": False, "frames": 2},
        # Dynamics: a stretch of constant-energy steps of the large box from a given state, and the state back.
        {"name": "md131072_mixed", "kind": "md", "system": "water", "n": 32, "form": "mixed", "strict": False, "steps": 10},
        # Constant-pressure dynamics of a small box: the cell, its link cells and k-vectors change every step.
        {"name": "npt864_mixed", "kind": "npt", "system": "water", "n": 6, "form": "mixed", "strict": False, "steps": 5},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["forces", "forces", "forces", "calls", "device", "device", "fit", "md", "npt"])
    form = rng.choice(["mixed", "mixed", "fp64"])
    if kind == "npt":
        return {"kind": kind, "system": "water", "n": rng.randint(5, 10), "form": form, "strict": False,
                "steps": rng.randint(2, 8)}
    if kind == "fit":
        return {"kind": kind, "system": "water", "n": rng.randint(5, 16 if form == "mixed" else 9), "form": form,
                "strict": rng.random() < 0.3, "frames": rng.randint(1, 4)}
    system = rng.choice(["argon", "water", "water", "mcy", "rocksalt", "wall"])
    if kind == "md":
        system = rng.choice(["argon", "water", "water"])
    n = {"argon": lambda: _log(rng, 4, 30), "water": lambda: _log(rng, 5, 32), "mcy": lambda: _log(rng, 5, 28),
         "rocksalt": lambda: _log(rng, 4, 22), "wall": lambda: rng.randint(6, 12)}[system]()
    case = {"kind": kind, "system": system, "n": n, "form": form, "strict": rng.random() < 0.4}
    if kind == "md":
        case["steps"] = rng.randint(2, 12)
        if form == "fp64" and system == "water":
            case["n"] = min(n, 20)
    return case


def _system(case, seed):
    k, n, strict = case["system"], case["n"], case["strict"]
    if k == "argon":
        return S.argon_fcc(ncell=n, seed=seed, strict=strict)
    if k == "water" or k == "mcy":
        return S.water(nside=n, seed=seed, strict=strict, model="mcy" if k == "mcy" else "tip4p")
    if k == "rocksalt":
        s = S.rock_salt(ncell=n, seed=seed)
        s.control.strict_cutoff = strict
        return s
    if k == "wall":
        return S.water_on_framework(nside=n, nlayers=n - 2, nwall=n + 1, seed=seed, strict=strict)
    raise ValueError(k)


def _fit_inputs(case, seed):
    """The water frames of a fit, its perturbed parameters and the reference forces under the original ones."""
    base = _system(case, seed)
    rng = np.random.default_rng(seed + 1000003)
    eps, sigma, q = rng.uniform(0.9, 1.1, 3)
    potpar = np.array(base.potpar, np.float64)
    potpar[1 + base.max_id, 0] *= eps
    potpar[1 + base.max_id, 1] *= sigma
    chg = base.chg() * q                      # neutral as before
    frames = water_frames(base, case["frames"], seed=seed + 7)
    return base, frames, potpar, chg


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fit":
        base, frames, potpar, chg = _fit_inputs(case, seed)
        refs = [np.ascontiguousarray(_Exact(f).forces()[0].cpu().numpy()) for f in frames]
        ff = ForceField(base, precision=case["form"])
        problem = FitProblem(ff, [f.site for f in frames], [f.c_of_m for f in frames], refs,
                             1.0 / (3 * base.nsites * len(frames)))
        return {"case": case, "ff": ff, "problem": problem, "potpar": torch.from_numpy(potpar),
                "chg": torch.from_numpy(chg), "alpha": torch.tensor(base.control.alpha, dtype=torch.float64)}
    sysm = _system(case, seed)
    ff = ForceField(sysm, precision=case["form"])
    st = {"case": case, "ff": ff, "sys": sysm}
    if kind == "device":
        st["stream"] = torch.cuda.Stream()
        ff.set_stream(st["stream"].cuda_stream)
        st["site"] = torch.from_numpy(np.ascontiguousarray(sysm.site)).cuda()
        st["force"] = torch.zeros_like(st["site"])
        st["record"] = torch.zeros(11, dtype=torch.float64, device="cuda")     # energies [2], stress [9]
    elif kind in ("md", "npt"):
        dyn = species_dynamics(sysm, 0.010 if case["system"] == "argon" else 0.001)
        st["start"] = thermal_state(sysm, dyn, 120.0 if case["system"] == "argon" else 300.0, seed + 17)
        if kind == "md":
            st["md"] = MolecularDynamics(ff, dyn, st["start"])
        else:
            st["dyn"] = dyn
    return st


def _record(pe, stress):
    """A step's energies and stress as the averages of a run take them: one record."""
    return np.concatenate([np.asarray(pe).reshape(-1), np.asarray(stress).reshape(-1)])


def _handed_on(case, arrays):
    """Results as the program keeps them: float64 of the FP64 form, float32 of the mixed form."""
    return arrays if case["form"] == "fp64" else [np.asarray(a, np.float32) for a in arrays]


def run(st):
    case, ff = st["case"], st["ff"]
    kind = case["kind"]
    if kind == "forces":
        f, pe, stress = ff.forces()
        return _handed_on(case, [f, _record(pe, stress)])
    if kind == "calls":
        f, pe_r, stress = ff.force_calc()
        f, pe_k, stress = ff.ewald(site_force=f, stress=stress)
        return _handed_on(case, [f, _record([pe_r, pe_k], stress)])
    if kind == "device":
        with torch.cuda.stream(st["stream"]):
            pe = st["record"].data_ptr()
            ff.forces_device(st["site"].data_ptr(), st["force"].data_ptr(), pe, pe + 16)
            out = [st["force"], st["record"]]
            return out if case["form"] == "fp64" else [t.float() for t in out]
    if kind == "fit":
        # the model's parameters; alpha is a numerical setting of the Ewald sum that a fit leaves alone
        leaves = [st[k].clone().requires_grad_(True) for k in ("potpar", "chg")]
        loss = ForceMatchLoss.apply(*leaves, st["alpha"], st["problem"])
        loss.backward()
        grad = torch.cat([t.grad.reshape(-1) for t in leaves])     # the flat vector an optimiser steps along
        out = [loss.detach().numpy(), grad.numpy()]
        return _handed_on(case, out)
    if kind == "md":
        st["md"].set_state(st["start"])
        e = st["md"].run(case["steps"])
        s = st["md"].state()
        return _handed_on(case, [e, s.c_of_m, s.mom, s.quat, s.amom])
    if kind == "npt":
        md = MolecularDynamics(ff, st["dyn"], st["start"])
        md.set_thermostat(300.0, 50.0)
        md.set_barostat(1, 0.0, 100.0)
        e = md.run(case["steps"])
        s = md.state()
        h, hmom = md.cell()
        return _handed_on(case, [e, s.c_of_m, s.mom, s.quat, s.amom, h, hmom])
    raise ValueError(kind)


def _counts(case):
    """(sites, charged sites, site pairs within the cut-off, k-vectors)"""
    k, n = case["system"], case["n"]
    if k == "argon":
        N, vol, rc, kc, nq = 4 * n ** 3, 4 * n ** 3 / 0.0213, 8.5, 0.0, 0
    elif k == "rocksalt":
        N, vol, rc, kc = 8 * n ** 3, (5.64 * n) ** 3, 10.0, S.ewald_k_cutoff(0.35)
        nq = N
    elif k == "wall":
        N, vol, rc, kc = 4 * n * n * (n - 2) + (n + 1) ** 2, (3.1 * n) ** 3, 9.0, S.ewald_k_cutoff(0.3)
        nq = N - n * n * (n - 2)
    else:
        N, vol, rc, kc = 4 * n ** 3, n ** 3 * 18.015 / 0.60221367, 9.0, S.ewald_k_cutoff(0.3)
        nq = 3 * n ** 3
    pairs = 0.5 * N * (N / vol) * 4.0 / 3.0 * math.pi * rc ** 3
    nk = 0.5 * 4.0 / 3.0 * math.pi * kc ** 3 * vol / (2 * math.pi) ** 3
    return N, nq, pairs, nk


def work(case):
    """Co-ordinates read and forces written once; per pair the 65 operations of the pair potential with the Ewald term,
    per charged site and k-vector 8 for the structure factor and 9 for the force."""
    N, nq, pairs, nk = _counts(case)
    one = 65.0 * pairs + 17.0 * nq * nk
    if case["kind"] == "fit":
        # forward, then again with the derivatives: three more weighted structure factors and a sum over k per site
        frames = case["frames"]
        return {"bytes": frames * (24.0 * N * 4 + 8.0 * N), "flops": frames * (2 * one + 65.0 * pairs + 40.0 * nq * nk)}
    if case["kind"] in ("md", "npt"):
        return {"bytes": 2 * 28.0 * N, "flops": case["steps"] * (one + 300.0 * N / 4)}
    return {"bytes": 48.0 * N, "flops": one}


# ---------------------------------------------------------------------------------------------------------------------
# What the results are in 64 bits: the definitions written out in torch, without this package's kernels or library.
_AS = (0.254829592, -0.284496736, 1.421413741, -1.453152027, 1.061405429)      # A&S 7.1.26, which defines the erfc term


def _erfc_as(x):
    t = 1.0 / (1.0 + 0.3275911 * x)
    return t * (_AS[0] + t * (_AS[1] + t * (_AS[2] + t * (_AS[3] + t * _AS[4])))) * torch.exp(-x * x)


def _pair(ptype, r2, qq, p, alpha):
    """(f, u) of each pair: f = -U'(r) / r."""
    rs = 1.0 / r2
    f = u = torch.zeros_like(r2)
    if ptype == S.LJPOT:
        s6 = (p[:, 1] * p[:, 1] * rs) ** 3
        u = p[:, 0] * (s6 * s6 - s6)
        f = rs * 6.0 * p[:, 0] * (2.0 * s6 * s6 - s6)
    elif ptype == S.E6POT:
        r = torch.sqrt(r2)
        e = p[:, 1] * torch.exp(-p[:, 2] * r)
        r6 = p[:, 0] * rs ** 3
        u, f = e - r6, -6.0 * rs * r6 + p[:, 2] * e / r
    elif ptype == S.MCYPOT:
        r = torch.sqrt(r2)
        e1, e2 = p[:, 0] * torch.exp(-p[:, 1] * r), -p[:, 2] * torch.exp(-p[:, 3] * r)
        u, f = e1 + e2, (p[:, 1] * e1 + p[:, 3] * e2) / r
    if float(alpha) > 0:
        r = torch.sqrt(r2)
        t = qq * _erfc_as(alpha * r) / r
        u = u + t
        f = f + rs * (t + qq * (2.0 / math.sqrt(math.pi)) * alpha * torch.exp(-(alpha * alpha) * r2))
    return f, u


class _Exact:
    """One configuration's energies, forces and stress from the definitions, on the GPU where there is one."""

    def __init__(self, sysm, potpar=None, chg=None):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        d = self._t
        self.sys, c = sysm, sysm.control
        self.h, self.N = np.asarray(sysm.h, np.float64), sysm.nsites
        self.hinv = np.linalg.inv(self.h)
        self.vol = float(np.linalg.det(self.h))
        self.x = d(np.ascontiguousarray(sysm.site.T))
        self.ids = torch.from_numpy(sysm.site_ids().astype(np.int64)).to(self.dev)
        self.mol = torch.from_numpy(sysm.molmap().astype(np.int64)).to(self.dev)
        self.potpar = d(np.asarray(sysm.potpar if potpar is None else potpar))
        self.chg = d(sysm.chg() if chg is None else chg)
        self.alpha = c.alpha
        nfw = sum(s.nsites * s.nmols for s in sysm.species if s.framework)
        self.fw = torch.arange(self.N, device=self.dev) >= self.N - nfw
        self._pairs = None

    def _t(self, a):
        return torch.from_numpy(np.array(a, np.float64)).to(self.dev)

    def pairs(self):
        """(i, j, r = x_j - x_i) of every evaluated pair: the link cells' (every site pair of cells whose origins are
        within the cut-off), or with the strict cut-off those within it."""
        if self._pairs is not None:
            return self._pairs
        c, h = self.sys.control, self.h
        sub = c.subcell if c.subcell > 0 else c.cutoff / 5.0
        n = np.array([int(h[k, k] / sub + 0.5) for k in range(3)])
        m = np.ceil(c.cutoff * n * np.linalg.norm(self.hinv, axis=1)).astype(int)
        if c.strict_cutoff:
            m = m + 2
        g = [np.arange(-(v - 1), v) for v in m]
        if not c.strict_cutoff:               # the reference's half list: x from 0, the others from -m
            g = [np.arange(-v, v) for v in m]
        o = np.stack(np.meshgrid(*g, indexing="ij"), -1).reshape(-1, 3)
        half = (o[:, 0] > 0) | ((o[:, 0] == 0) & (o[:, 1] > 0)) | ((o[:, 0] == 0) & (o[:, 1] == 0) & (o[:, 2] >= 0))
        o = o[half]
        if not c.strict_cutoff:
            o = o[(((o / n) @ h.T) ** 2).sum(1) < c.cutoff ** 2]
        dev = self.dev
        nt = torch.from_numpy(n).to(dev)
        s = self.x @ self._t(self.hinv).T
        cell = torch.minimum(torch.floor((s + 0.5) * nt).long().clamp(min=0), nt - 1)
        cid = cell[:, 2] + n[2] * (cell[:, 1] + n[1] * cell[:, 0])
        order = torch.argsort(cid, stable=True)
        start = torch.searchsorted(cid[order].contiguous(), torch.arange(int(np.prod(n)) + 1, device=dev))
        ht, out = self._t(h), []
        for k in range(0, len(o), 16):
            d = torch.from_numpy(o[k:k + 16]).to(dev)
            p = cell[:, None, :] + d[None]
            img = torch.div(p, nt, rounding_mode="floor")
            p = p - img * nt
            q = (p[..., 2] + n[2] * (p[..., 1] + n[1] * p[..., 0])).reshape(-1)
            cnt = start[q + 1] - start[q]
            row = torch.repeat_interleave(torch.arange(q.numel(), device=dev), cnt)
            first = torch.cumsum(cnt, 0) - cnt
            j = order[start[q][row] + torch.arange(row.numel(), device=dev) - first[row]]
            i = torch.div(row, d.shape[0], rounding_mode="floor")
            keep = (d != 0).any(1)[row % d.shape[0]] | (i < j)
            keep &= ~(self.fw[i] & self.fw[j])
            i, j, im = i[keep], j[keep], img.reshape(-1, 3)[row[keep]]
            r = self.x[j] - self.x[i] + im.double() @ ht.T
            if c.strict_cutoff:
                near = (r * r).sum(1) <= c.cutoff ** 2
                i, j, r = i[near], j[near], r[near]
            out.append((i, j, r))
        self._pairs = tuple(torch.cat(v) for v in zip(*out))
        return self._pairs

    def kvectors(self):
        """(integer triples, k, the energy prefactor, the stress factor) of the half sphere."""
        c, h = self.sys.control, self.h
        top = np.floor(c.k_cutoff / (2 * math.pi) * np.linalg.norm(h, axis=0)).astype(int)
        o = np.stack(np.meshgrid(*[np.arange(-v, v + 1) for v in top], indexing="ij"), -1).reshape(-1, 3)
        half = (o[:, 0] > 0) | ((o[:, 0] == 0) & (o[:, 1] > 0)) | ((o[:, 0] == 0) & (o[:, 1] == 0) & (o[:, 2] > 0))
        o = o[half]
        k = 2 * math.pi * o @ self.hinv
        k2 = (k * k).sum(1)
        o, k, k2 = o[k2 < c.k_cutoff ** 2], k[k2 < c.k_cutoff ** 2], k2[k2 < c.k_cutoff ** 2]
        a = self.alpha
        coeff = 8 * math.pi / self.vol * np.exp(-k2 / (4 * a * a)) / k2
        return self._t(o), self._t(k), self._t(coeff), self._t(2 * (1 + k2 / (4 * a * a)) / k2)

    def _waves(self):
        """Per run of k-vectors: (k, prefactor, stress factor, cos, sin of k.r over the charged sites)."""
        n, k, coeff, coeff2 = self.kvectors()
        on = self.chg != 0
        s = (self.x @ self._t(self.hinv).T)[on]
        step = max(1, (1 << 25) // max(1, int(on.sum())))
        for a in range(0, len(k), step):
            ph = n[a:a + step] @ s.T
            ph = 2 * math.pi * (ph - torch.floor(ph))
            yield k[a:a + step], coeff[a:a + step], coeff2[a:a + step], torch.cos(ph), torch.sin(ph)

    def forces(self):
        """(force [3, N], pe [2], stress [9])"""
        i, j, r = self.pairs()
        F = torch.zeros_like(self.x)
        pe, st = torch.zeros(2, dtype=torch.float64, device=self.dev), torch.zeros(9, dtype=torch.float64, device=self.dev)
        M = self.sys.max_id
        up = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]
        for a in range(0, len(i), 1 << 22):
            ii, jj, rr = i[a:a + (1 << 22)], j[a:a + (1 << 22)], r[a:a + (1 << 22)]
            f, u = _pair(self.sys.ptype, (rr * rr).sum(1), self.chg[ii] * self.chg[jj],
                         self.potpar[self.ids[ii] * M + self.ids[jj]], self.alpha)
            w = f[:, None] * rr
            F.index_add_(0, ii, -w)
            F.index_add_(0, jj, w)
            # a molecule's own pairs: their energy is what the intramolecular correction takes off again
            pe[0] += u[(self.mol[ii] != self.mol[jj]) | self.fw[ii]].sum()
            for x, y in up:
                st[3 * x + y] += (w[:, x] * rr[:, y]).sum()
        if self.alpha > 0:
            on = self.chg != 0
            q, fw = self.chg[on], self.fw[on]
            Fk = torch.zeros(3, len(q), dtype=torch.float64, device=self.dev)
            qf = torch.where(fw, q, torch.zeros_like(q))
            for k, cf, cf2, c, s in self._waves():
                C, Sn, Cf, Sf = c @ q, s @ q, c @ qf, s @ qf
                e = 0.5 * cf * ((C * C + Sn * Sn) - (Cf * Cf + Sf * Sf))
                pe[1] += e.sum()
                for x, y in up:
                    st[3 * x + y] += (e * (1.0 if x == y else 0.0) - e * cf2 * k[:, x] * k[:, y]).sum()
                Fk += ((k.T * (cf * C)) @ s - (k.T * (cf * Sn)) @ c)
                if bool(fw.any()):
                    Fk[:, fw] -= ((k.T * (cf * Cf)) @ s[:, fw] - (k.T * (cf * Sf)) @ c[:, fw])
            F[on] += (q * Fk).T
            self_e, sheet = self._self_sheet()
            pe[1] += -self_e + sheet / self.vol
            for d in range(3):
                st[4 * d] += sheet / self.vol
        return F.T.contiguous(), pe, st

    def _self_sheet(self):
        a, q0, chg = self.alpha, 0, self.chg.cpu().numpy()
        e, qnf, qfw = 0.0, 0.0, 0.0
        for sp in self.sys.species:
            q = chg[q0:q0 + sp.nsites * sp.nmols]
            q0 += len(q)
            if sp.framework:
                qfw += q.sum()
                continue
            qnf += q.sum()
            e += a / math.sqrt(math.pi) * float((q * q).sum())
            p = np.asarray(sp.p_f_sites)
            for m in range(sp.nsites):
                for n in range(m + 1, sp.nsites):
                    d = float(np.linalg.norm(p[m] - p[n]))
                    e += sp.nmols * q[m] * q[n] * (1.0 - float(_erfc_as(torch.tensor(a * d, dtype=torch.float64)))) / d
        sheet = math.pi * qfw ** 2 / (2 * a * a)
        if abs(qnf + qfw) * S.CONV_Q > 1e-5:
            sheet -= math.pi * (qnf + qfw) ** 2 / (2 * a * a)
        return e, sheet

    def fit(self, f_ref, weight):
        """Loss weight * sum |F - F_ref|^2 and its gradient by the table and the charges."""
        F = self.forces()[0]
        v = F - self._t(f_ref)
        loss = weight * float((v * v).sum())
        v = (2 * weight * v).T.contiguous()
        pot, chg = self.potpar.clone().requires_grad_(True), self.chg.clone().requires_grad_(True)
        i, j, r = self.pairs()
        M = self.sys.max_id
        for a in range(0, len(i), 1 << 20):
            ii, jj, rr = i[a:a + (1 << 20)], j[a:a + (1 << 20)], r[a:a + (1 << 20)]
            r2, qq = (rr * rr).sum(1), chg[ii] * chg[jj]
            # the force on a site reads the table at [its identifier][the partner's]
            fi = _pair(self.sys.ptype, r2, qq, pot[self.ids[ii] * M + self.ids[jj]], self.alpha)[0]
            fj = _pair(self.sys.ptype, r2, qq, pot[self.ids[jj] * M + self.ids[ii]], self.alpha)[0]
            (fj * (v[jj] * rr).sum(1) - fi * (v[ii] * rr).sum(1)).sum().backward()
        gq = chg.grad.clone()
        n, kk, cf_all, _ = self.kvectors()
        s_all = self.x @ self._t(self.hinv).T
        step = max(1, (1 << 25) // self.N)
        for a in range(0, len(kk), step):
            k, cf = kk[a:a + step], cf_all[a:a + step]
            ph = n[a:a + step] @ s_all.T
            ph = 2 * math.pi * (ph - torch.floor(ph))
            c, s = torch.cos(ph), torch.sin(ph)
            kv = k @ v.T
            C, Sn = c @ self.chg, s @ self.chg
            Tc, Ts = (c * kv) @ self.chg, (s * kv) @ self.chg
            gq += (cf * Ts) @ c - (cf * Tc) @ s + ((cf * C)[:, None] * s * kv - (cf * Sn)[:, None] * c * kv).sum(0)
        return loss, np.concatenate([pot.grad.cpu().numpy().reshape(-1), gq.cpu().numpy()])


def exact(case, seed):
    kind = case["kind"]
    if kind in ("forces", "calls", "device"):
        f, pe, st = (t.cpu().numpy() for t in _Exact(_system(case, seed)).forces())
        return [f, _record(pe, st)]
    if kind == "fit":
        base, frames, potpar, chg = _fit_inputs(case, seed)
        w = 1.0 / (3 * base.nsites * len(frames))
        loss, grad = 0.0, 0.0
        for f in frames:
            ref = _Exact(f).forces()[0].cpu().numpy()
            a, g = _Exact(f, potpar, chg).fit(ref, w)
            loss, grad = loss + a, grad + g
        return [np.array(loss), grad]
    return None          # a trajectory: a hundred and more such evaluations per pass with the equations of motion between
