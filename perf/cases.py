"""The work that programs have this package do, as measurable cases.

A case is one pass through the public entry points on one synthetic system
(the recipe of ``ad_afqmc_b200/synthetic.py``, drawn on the GPU from the seed),
with walkers spread around the trial determinant.  ``path`` names the entry
point:

  sampler   ``sampler.propagate_phaseless``: a driver's energy block, launched
            call by call (fields, steps, QR, energies, comb)
  graph     ``BlockGraph.replay``: the same block recorded once and replayed,
            as the server does; with ``lno`` the fragment's orbital energy too
  batch     ``GroupedBatchGraph.replay``: one block of several fragments of
            different sizes (N ~ U[30,160], No = N/4, G ~ U[4N,6N], W ~ U[64,256])
  step      ``propagator_afqmc.propagate_constrained``: one phaseless step
  energy    ``trial.calc_energy`` on the propagator's engine
  setup     what a solve pays before its first step: both sets of
            intermediates, initial walkers, their energy and overlaps
"""

import math
import random

import numpy as np
import torch

from ad_afqmc_b200 import hamiltonian, propagation, sampling, wavefunctions
from ad_afqmc_b200.graphs import BlockGraph, GroupedBatchGraph
from ad_afqmc_b200.walkers import RHFWalkers, UHFWalkers

DT = 0.005
N_EXP = 6
F64, C128 = torch.float64, torch.complex128


def _case(name, path, trial, norb, na, nb, nchol, walkers, precision, **more):
    return dict(name=name, path=path, trial=trial, norb=norb, na=na, nb=nb, nchol=nchol,
                walkers=walkers, precision=precision, **more)


def listed():
    return [
        # the smallest solve: the FCIDUMP of the driver test (6 orbitals, 3+3 electrons, 15
        # Cholesky vectors, 50 walkers, UHF), in the default precision; launches count
        _case("block_n6_uhf_fp64", "sampler", "uhf", 6, 3, 3, 15, 50, "fp64", steps=10),
        # the N = 10 workload (a ten-atom chain in a minimal basis), recorded
        _case("graph_n10_rhf_fp64", "graph", "rhf", 10, 5, 5, 50, 100, "fp64", steps=10),
        # an ordinary molecule in the default precision, odd sizes, called as the driver does
        _case("block_n95_rhf_fp64", "sampler", "rhf", 95, 23, 23, 471, 161, "fp64", steps=10),
        # a batch of local-correlation fragments of uneven sizes
        _case("batch8_mixed", "batch", "rhf", 0, 0, 0, 0, 0, "mixed", steps=10, fragments=8, shapes=1004),
        # one large fragment, served alone from its recorded block
        _case("graph_n157_rhf_mixed", "graph", "rhf", 157, 39, 39, 863, 231, "mixed", steps=10),
        # an LNO fragment: every block averages the orbital energy too
        _case("graph_n100_lno_mixed", "graph", "rhf", 100, 25, 25, 500, 128, "mixed", steps=10, lno=True),
        # the benchmark workload, step and energy, in both precisions
        _case("step_n200_rhf_mixed", "step", "rhf", 200, 40, 40, 1000, 512, "mixed"),
        _case("energy_n200_rhf_mixed", "energy", "rhf", 200, 40, 40, 1000, 512, "mixed"),
        _case("step_n200_rhf_fp64", "step", "rhf", 200, 40, 40, 1000, 512, "fp64"),
        _case("energy_n200_rhf_fp64", "energy", "rhf", 200, 40, 40, 1000, 512, "fp64"),
        # set-up of the largest served fragment
        _case("setup_n250_rhf_mixed", "setup", "rhf", 250, 62, 62, 1250, 256, "mixed"),
        # the largest workload: open shell, unrestricted walkers, a whole recorded block
        _case("graph_n300_uhf_mixed", "graph", "uhf", 300, 60, 58, 1500, 1024, "mixed", steps=10),
    ]


def draw(rng):
    """One more case: the same paths, sizes spread over their logarithm."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    path = rng.choice(["sampler", "graph", "graph", "batch", "step", "energy", "setup"])
    precision = rng.choice(["fp64", "mixed", "mixed"])
    steps = rng.randint(5, 12)
    if path == "batch":
        return dict(path=path, trial="rhf", norb=0, na=0, nb=0, nchol=0, walkers=0, precision="mixed",
                    steps=steps, fragments=rng.randint(3, 10), shapes=rng.randrange(1 << 20))
    # a lone step or energy is called on systems where it takes a while; FP64 blocks end at
    # the benchmark size so that no pass costs more than the largest listed one
    lo, hi = {"sampler": (6, 200), "graph": (6, 300), "step": (90, 300), "energy": (40, 300),
              "setup": (30, 250)}[path]
    if precision == "fp64":
        hi = min(hi, 200)
    norb = size(lo, hi)
    if path == "setup":
        norb += norb % 2  # the second spin's density matrix of an odd norb is not 16-byte aligned: refused
    trial = rng.choice(["rhf", "rhf", "uhf"])
    na = max(2, min(62, int(round(norb * rng.uniform(0.18, 0.5 if norb < 30 else 0.26)))))
    nb = na if trial == "rhf" else max(1, na - rng.randint(0, 2))
    nchol = int(round(norb * rng.uniform(2.5, 6.0) if norb < 30 else norb * rng.uniform(4.0, 5.5)))
    c = dict(path=path, trial=trial, norb=norb, na=na, nb=nb, nchol=nchol,
             walkers=size(48, 384 if precision == "fp64" else 512 if norb <= 200 else 768), precision=precision)
    if path in ("sampler", "graph"):
        c["steps"] = steps
    if path == "graph" and trial == "rhf" and rng.random() < 0.25:
        c["lno"] = True
    if path in ("step", "energy") and precision == "mixed" and rng.random() < 0.2:
        c["precision"] = "mixed_hi"
    return c


def _fragments(case):
    """The solves of a case: itself, or the fragments of a batch."""
    if case["path"] != "batch":
        return [case]
    r = random.Random(case["shapes"])
    out = []
    for _ in range(case["fragments"]):
        n = r.randint(30, 160)
        no = int(round(n / 4))
        out.append(dict(case, norb=n, na=no, nb=no, nchol=r.randint(4 * n, 6 * n), walkers=r.randint(64, 256)))
    return out


# ---------------------------------------------------------------------------
# inputs (torch only: the 64-bit statement below starts from the same ones)
# ---------------------------------------------------------------------------
def _inputs(case, seed):
    n, g, w = case["norb"], case["nchol"], case["walkers"]
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)

    def normal(*shape):
        return torch.randn(*shape, dtype=F64, device=dev, generator=gen)

    def symmetric(a):
        u = torch.triu(a)
        return u + torch.triu(u, 1).transpose(-1, -2)

    # Cholesky vectors at a scale where the population lives
    scale = 0.5 if n < 30 else 0.1
    decay = torch.exp(-torch.arange(g, dtype=F64, device=dev) / n) * (scale / math.sqrt(n))
    chol = symmetric(normal(g, n, n)) * decay.reshape(-1, 1, 1)
    h1 = 0.1 * symmetric(normal(n, n)) + torch.diag(torch.linspace(-3.0, 1.0, n, dtype=F64, device=dev))
    h1 = torch.stack([h1, h1])
    r = symmetric(normal(n, n))
    nocc = [case["na"], case["nb"]]
    if case["trial"] == "rhf":
        mo = [torch.linalg.eigh(h1[0].cpu())[1][:, : nocc[0]].contiguous().to(dev)] * 2
    else:
        mo = [torch.linalg.eigh((h1[s] + sg * 0.05 * r).cpu())[1][:, : nocc[s]].contiguous().to(dev)
              for s, sg in ((0, 1.0), (1, -1.0))]
    sectors = 1 if case["trial"] == "rhf" else 2
    walkers = []
    for s in range(sectors):
        eps = 0.15 / math.sqrt(nocc[s])
        walkers.append(torch.complex(mo[s] + eps * normal(w, n, nocc[s]), eps * normal(w, n, nocc[s])))
    prj = normal(1, nocc[0])
    return dict(chol=chol.reshape(g, n * n), h1=h1, mo=mo, walkers=walkers, prj=prj / prj.norm(),
                fields=normal(w, g), rdm1=torch.stack([mo[0] @ mo[0].T, mo[1] @ mo[1].T]))


def _solve(case, seed):
    """A solve as a program sets it up: trial, integrals, propagator, walkers."""
    x = _inputs(case, seed)
    nelec = (case["na"], case["nb"])
    wave = {"rdm1": x["rdm1"], "mo_coeff": x["mo"][0] if case["trial"] == "rhf" else list(x["mo"])}
    if case.get("lno"):
        trial = wavefunctions.rhf_lno(case["norb"], nelec)
        wave["prjlo"] = x["prj"]
    else:
        trial = (wavefunctions.rhf if case["trial"] == "rhf" else wavefunctions.uhf)(case["norb"], nelec)
    s = dict(case=case, seed=seed, trial=trial, wave=wave, ham=hamiltonian.hamiltonian(case["norb"]),
             raw={"h0": 0.0, "ene0": 0.0, "h1": x["h1"], "chol": x["chol"]}, fields=x["fields"])
    s["prop"] = propagation.propagator_afqmc(
        dt=DT, n_walkers=case["walkers"], n_exp_terms=N_EXP, precision=case["precision"],
        walker_type="restricted" if case["trial"] == "rhf" else "unrestricted")
    if case["path"] == "setup":
        return s
    hd = s["ham"].build_measurement_intermediates(dict(s["raw"]), trial, wave)
    s["hd"] = s["ham"].build_propagation_intermediates(hd, s["prop"], trial, wave)
    own = [t.clone() for t in x["walkers"]]
    s["pd"] = s["prop"].init_prop_data(trial, wave, s["hd"], seed=seed,
                                       init_walkers=RHFWalkers(own[0]) if len(own) == 1 else UHFWalkers(own))
    return s


def _record(s):
    return BlockGraph(s["ham"], s["hd"], s["prop"], s["trial"], s["wave"], s["pd"],
                      n_prop_steps=s["case"]["steps"], lno=bool(s["case"].get("lno")))


def _kept(pd):
    w = pd["walkers"].data
    own = list(w) if isinstance(w, list) else [w]
    return [own[i].clone() for i in range(len(own))] + [pd["weights"].clone(), pd["overlaps"].clone(),
                                                        pd["_scalars"].clone()]


def _rewind(bg, kept):
    """Back to the initial population after the recording's warm-up block."""
    for t, u in zip(bg.tensors + [bg.pd["weights"], bg.pd["overlaps"], bg.pd["_scalars"]], kept):
        t.copy_(u)
    bg.counter.zero_()


def prepare(case, seed):
    solves = [_solve(c, seed + 7919 * i) for i, c in enumerate(_fragments(case))]
    if case["path"] not in ("graph", "batch"):
        s = solves[0]
        if case["path"] == "sampler":
            s["sampler"] = sampling.sampler(n_prop_steps=case["steps"], n_ene_blocks=1, n_sr_blocks=1)
        elif case["path"] == "energy":
            s["engine"] = s["prop"].engine(s["hd"], s["trial"], s["wave"])
        return s
    kept = [_kept(s["pd"]) for s in solves]
    blocks = [_record(s) for s in solves]
    whole = blocks[0] if case["path"] == "graph" else GroupedBatchGraph(blocks)
    whole.capture(warmup=1)
    for bg, k in zip(blocks, kept):
        _rewind(bg, k)
    return dict(case=case, solves=solves, blocks=blocks, whole=whole)


def _population(pd):
    return {"walkers": pd["walkers"].data, "weights": pd["weights"], "overlaps": pd["overlaps"]}


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "graph" or path == "batch":
        state["whole"].replay()
        return [dict(_population(bg.pd), block=bg.block_out) for bg in state["blocks"]]
    s = state
    if path == "sampler":
        e, s["pd"] = s["sampler"].propagate_phaseless(s["ham"], s["hd"], s["prop"], s["pd"], s["trial"], s["wave"])
        return dict(_population(s["pd"]), energy=e)
    if path == "step":
        s["pd"] = s["prop"].propagate_constrained(s["trial"], s["hd"], s["pd"], s["fields"], s["wave"])
        return _population(s["pd"])
    if path == "energy":
        return s["trial"].calc_energy(s["pd"]["walkers"], s["hd"], s["wave"], engine=s["engine"])
    # set-up; the initial walkers themselves are fixed up to a rotation among equally occupied
    # orbitals only, so their energy and the moduli of their overlaps stand for them
    wave = {k: s["wave"][k] for k in ("rdm1", "mo_coeff")}
    hd = s["ham"].build_measurement_intermediates(dict(s["raw"]), s["trial"], wave)
    hd = s["ham"].build_propagation_intermediates(hd, s["prop"], s["trial"], wave)
    pd = s["prop"].init_prop_data(s["trial"], wave, hd, seed=s["seed"])
    return {"h1": hd["h1"], "rot_h1": hd["rot_h1"], "rot_chol": hd["rot_chol"], "mf_shifts": hd["mf_shifts"],
            "h0_prop": hd["h0_prop"], "exp_h1": hd["exp_h1"], "e_estimate": pd["e_estimate"],
            "overlaps": torch.abs(pd["overlaps"])}


def work(case):
    """What a pass cannot do without: real operations of the contractions, and
    each operand (the Hamiltonian in the precision it is used in) read once and
    each result written once."""
    flops = bytes_ = 0.0
    for c in _fragments(case):
        n, g, w = c["norb"], c["nchol"], c["walkers"]
        occ = [c["na"]] if c["trial"] == "rhf" else [c["na"], c["nb"]]
        item = {"fp64": 8, "mixed": 4, "mixed_hi": 6}[c["precision"]]
        walker = 16.0 * w * n * sum(occ)
        chol, rot = float(item) * g * n * n, float(item) * g * n * sum(occ)
        step = energy = qr = 0.0
        for o in occ:
            step += 4.0 * g * n * o + 8.0 * (N_EXP - 1) * n * n * o + 8.0 * n * n * o + 16.0 * n * o * o + 16.0 * o ** 3
            energy += 4.0 * g * o * o * n + 8.0 * g * o * o + 12.0 * n * o * o + 8.0 * o ** 3
            qr += 8.0 * (2.0 * n * o * o - 2.0 / 3.0 * o ** 3)
        step += 4.0 * g * n * n
        if c["path"] == "step":
            flops += w * step
            bytes_ += 2 * walker + chol + rot + 8.0 * w * g
        elif c["path"] == "energy":
            flops += w * energy
            bytes_ += walker + rot + 16.0 * w
        elif c["path"] == "setup":
            flops += sum(2.0 * g * n * n * o for o in occ) + 2.0 * g * n ** 3 + 60.0 * n ** 3 + w * energy
            bytes_ += 8.0 * g * n * n + 8.0 * g * n * sum(occ) + walker + chol
        else:
            flops += w * (c["steps"] * step + energy + qr)
            bytes_ += c["steps"] * (2 * walker + chol + rot + 8.0 * w * g) + rot + 4 * walker
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------------------
# the same passes in 64 bits, in plain torch and numpy
# ---------------------------------------------------------------------------
def _philox(seed, counters, third):
    """Philox4x32-10 of (counter, third, 0) under the 64-bit seed: four uint32 words."""
    m = np.uint64(0xFFFFFFFF)
    sh = np.uint64(32)
    c0, c1 = counters & m, counters >> sh
    c2, c3 = np.full_like(counters, third), np.zeros_like(counters)
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c0, np.uint64(0xCD9E8D57) * c2
        c0, c1, c2, c3 = (p1 >> sh) ^ c1 ^ np.uint64(k0), p1 & m, (p0 >> sh) ^ c3 ^ np.uint64(k1), p0 & m
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c0, c1, c2, c3


def _unit(hi, lo):
    return ((((hi << np.uint64(32)) | lo) >> np.uint64(11)).astype(np.float64) + 0.5) * 2.0 ** -53


def _normals(seed, n, dev):
    """The device's field stream: Box-Muller pairs of Philox blocks 0, 1, ..."""
    pairs = (n + 1) // 2
    out = torch.empty(2 * pairs, dtype=F64, device=dev)
    for a in range(0, pairs, 1 << 20):
        r = _philox(seed, np.arange(a, min(pairs, a + (1 << 20)), dtype=np.uint64), 0)
        u1, u2 = (torch.from_numpy(_unit(r[2 * i], r[2 * i + 1])).to(dev) for i in (0, 1))
        rad, ang = torch.sqrt(-2.0 * torch.log(u1)), 2.0 * math.pi * u2
        out[2 * a:2 * (a + u1.numel())] = torch.stack([rad * torch.cos(ang), rad * torch.sin(ang)], 1).reshape(-1)
    return out[:n], pairs


class _Plain:
    """One solve, every quantity in float64 / complex128."""

    def __init__(self, case, seed):
        x = _inputs(case, seed)
        self.case, self.x, self.seed = case, x, seed
        n, g = case["norb"], case["nchol"]
        self.rhf = case["trial"] == "rhf"
        self.mo = x["mo"][:1] if self.rhf else x["mo"]
        self.L = x["chol"].reshape(g, n, n)
        self.h1 = (x["h1"] + x["h1"].transpose(1, 2)) / 2.0
        h = [(self.h1[0] + self.h1[1]) / 2.0] if self.rhf else [self.h1[0], self.h1[1]]
        self.rot_h1 = [c.T @ a for c, a in zip(self.mo, h)]
        self.rot_chol = [torch.matmul(c.T, self.L) for c in self.mo]
        rdm = x["rdm1"][0] + x["rdm1"][1]
        mf = torch.einsum("gij,ij->g", self.L, rdm)
        self.mf = 1j * mf
        self.h0_prop = -torch.sum(self.mf ** 2) / 2.0
        v0 = torch.zeros(n, n, dtype=F64, device=mf.device)
        for a in range(0, g, 64):
            v0 += 0.5 * torch.matmul(self.L[a:a + 64], self.L[a:a + 64]).sum(0)
        v1 = torch.einsum("g,gij->ij", -mf, self.L)
        self.exp_h1 = [torch.linalg.matrix_exp(-DT / 2.0 * (a - v0 - v1)) for a in h]

    def green(self, walkers):
        """(W, N, No) W (C^T W)^-1 and the determinants, per sector."""
        th, det = [], []
        for w, c in zip(walkers, self.mo):
            s = torch.matmul(c.T.to(C128), w)
            th.append(torch.linalg.solve(s.transpose(1, 2), w.transpose(1, 2)).transpose(1, 2))
            det.append(torch.linalg.det(s))
        return th, (det[0] * det[0] if self.rhf else det[0] * det[1])

    def force_bias(self, th):
        f = 0.0
        for t, rc in zip(th, self.rot_chol):
            m = rc.reshape(rc.shape[0], -1)
            flat = t.transpose(1, 2).reshape(t.shape[0], -1)
            f = f + torch.complex(flat.real @ m.T, flat.imag @ m.T)
        return 2.0 * f if self.rhf else f

    def energy(self, th, orbital=False):
        w, g = th[0].shape[0], self.L.shape[0]
        e1, cs, exc, orb = 0.0, 0.0, 0.0, 0.0
        for t, rh, rc in zip(th, self.rot_h1, self.rot_chol):
            o = t.shape[2]
            e1 = e1 + torch.einsum("jp,wpj->w", rh.to(C128), t)
            c = torch.empty(w, g, dtype=C128, device=t.device)
            x = torch.zeros(w, dtype=C128, device=t.device)
            orb = torch.zeros(w, dtype=C128, device=t.device)
            step = max(1, int(2 ** 26 // (g * o * o)))
            a = rc.reshape(g * o, -1)
            for i in range(0, w, step):
                b = torch.view_as_real(t[i:i + step]).permute(1, 0, 2, 3).reshape(t.shape[1], -1)
                f = torch.view_as_complex((a @ b).reshape(g, o, -1, o, 2).permute(2, 0, 1, 3, 4).contiguous())
                c[i:i + step] = torch.einsum("wgii->wg", f)
                x[i:i + step] = torch.einsum("wgij,wgji->w", f, f)
                if orbital:  # the virtual rows of Theta alone
                    p = self.x["prj"][0].to(C128)
                    b = torch.view_as_real(t[i:i + step, o:]).permute(1, 0, 2, 3).reshape(t.shape[1] - o, -1)
                    f = torch.view_as_complex((rc[:, :, o:].reshape(g * o, -1) @ b).reshape(g, o, -1, o, 2).permute(2, 0, 1, 3, 4).contiguous())
                    u, v = torch.einsum("i,wgij->wgj", p, f), torch.einsum("wgij,j->wgi", f, p)
                    orb[i:i + step] = (2.0 * torch.einsum("wgii->wg", f) * torch.einsum("wgj,j->wg", u, p)
                                       - torch.einsum("wgj,wgj->wg", u, v)).sum(1)
            cs, exc = cs + c, exc + x
        j = torch.sum(cs * cs, 1)
        e = 2.0 * j - exc + 2.0 * e1 if self.rhf else 0.5 * (j - exc) + e1
        return (e, orb) if orbital else e

    def step(self, p, fields):
        sdt = math.sqrt(DT)
        th, _ = self.green(p["walkers"])
        fs = -sdt * (1j * self.force_bias(th) - self.mf)
        x = fields - fs
        shift = torch.sum(x * self.mf, 1)
        term = torch.sum(fields * fs - fs * fs / 2.0, 1)
        w, n = x.shape[0], self.L.shape[1]
        m = self.L.reshape(self.L.shape[0], -1)
        v = (1j * sdt) * torch.complex(x.real @ m, x.imag @ m).reshape(w, n, n)
        new = []
        for t, e in zip(p["walkers"], self.exp_h1):
            y = torch.matmul(e.to(C128), t)
            out, z = y.clone(), y
            for k in range(1, N_EXP):
                z = torch.matmul(v, z) / k
                out += z
            new.append(torch.matmul(e.to(C128), out))
        p["walkers"] = new
        _, ov = self.green(new)
        ratio = ov / p["overlaps"]
        imp = torch.exp(-sdt * shift + term + DT * (p["shift"] + self.h0_prop)) * ratio
        ipl = torch.abs(imp) * torch.cos(torch.angle(torch.exp(-sdt * shift) * ratio))
        ipl = torch.where(torch.isnan(ipl) | (ipl < 1e-3) | (ipl > 100.0), torch.zeros_like(ipl), ipl)
        wt = ipl * p["weights"]
        p["weights"] = torch.where(wt > 100.0, torch.zeros_like(wt), wt)
        p["shift"] = p["e_estimate"] - 0.1 * torch.log(torch.sum(p["weights"]) / w) / DT
        p["overlaps"] = ov

    def start(self):
        th, ov = self.green(self.x["walkers"])
        e = torch.mean(self.energy(th).real)
        w = self.x["walkers"][0].shape[0]
        return {"walkers": list(self.x["walkers"]), "overlaps": ov, "e_estimate": e, "shift": e,
                "weights": torch.ones(w, dtype=F64, device=e.device)}

    def block(self):
        """One energy block and its comb; the fields and zeta of the path's own stream."""
        c, p = self.case, self.start()
        dev = p["weights"].device
        w = c["walkers"]
        f, used = _normals(self.seed, c["steps"] * w * c["nchol"], dev)
        for x in f.reshape(c["steps"], w, c["nchol"]):
            self.step(p, x)
        for s, t in enumerate(p["walkers"]):
            q, r = (a.to(dev) for a in torch.linalg.qr(t.cpu()))  # Householder, LAPACK's signs
            if not self.rhf:
                d = torch.prod(torch.sign(torch.diagonal(r, dim1=1, dim2=2).real), 1)
                q[:, :, 0] *= d.reshape(-1, 1)
            p["walkers"][s] = q
        th, ov = self.green(p["walkers"])
        lno = bool(c.get("lno"))
        e, orb = self.energy(th, True) if lno else (self.energy(th), None)
        ref = p["shift"] if lno else p["e_estimate"]
        e = torch.where(torch.abs(e.real - ref) > math.sqrt(2.0 / DT), ref, e.real)
        total = torch.sum(p["weights"])
        block = [torch.sum(e * p["weights"]) / total, total]
        if lno:
            block.append(torch.sum(orb.real * p["weights"]) / total)
        if c["path"] == "sampler":
            zeta = float(np.random.default_rng([self.seed, used, 0x5A5A]).random())
        else:
            r = _philox(self.seed, np.array([used], dtype=np.uint64), 1)
            zeta = float(_unit(r[0], r[1])[0])
        cum = np.cumsum(p["weights"].cpu().numpy())
        idx = np.minimum(np.searchsorted(cum, cum[-1] * (np.arange(w) + zeta) / w), w - 1)
        at = torch.from_numpy(idx).to(dev)
        out = {"weights": torch.full_like(p["weights"], float(cum[-1]) / w)}
        # in reduced precision a comb tooth may fall on the neighbouring walker
        alike = c["precision"] == "fp64"
        out["walkers"] = (([t[at] for t in p["walkers"]] if not self.rhf else p["walkers"][0][at]) if alike else None)
        out["overlaps"] = ov[at] if alike else None
        if c["path"] == "sampler":
            out["energy"] = block[0]
        else:
            out["block"] = torch.stack(block)
        return out


def exact(case, seed):
    path = case["path"]
    if path in ("graph", "batch"):
        return [_Plain(c, seed + 7919 * i).block() for i, c in enumerate(_fragments(case))]
    p = _Plain(case, seed)
    if path == "sampler":
        return p.block()
    if path == "energy":
        return p.energy(p.green(p.x["walkers"])[0])
    if path == "step":
        q = p.start()
        p.step(q, p.x["fields"])
        return {"walkers": q["walkers"][0] if p.rhf else q["walkers"], "weights": q["weights"],
                "overlaps": q["overlaps"]}
    one = lambda v: v[0] if p.rhf else v  # noqa: E731
    trial = [c.to(C128).unsqueeze(0) for c in p.mo]
    return {"h1": p.h1, "rot_h1": one(p.rot_h1), "rot_chol": one(p.rot_chol), "mf_shifts": p.mf,
            "h0_prop": p.h0_prop, "exp_h1": p.exp_h1[0] if p.rhf else torch.stack(p.exp_h1),
            "e_estimate": p.energy(p.green(trial)[0])[0].real,
            "overlaps": torch.ones(case["walkers"], dtype=F64, device=p.mf.device)}
