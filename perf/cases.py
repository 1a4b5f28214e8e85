"""Performance cases of the three- and four-phonon scattering path.

Each case is one call, or one short sequence of calls, that a user of the package makes
through its public entry points:

  solve    ScatteringRates.generate and .kappa on an open context (the body of a run over
           temperatures, smearings, samples or force constants)
  program  the whole thermal_conductivity sequence from the infile.* files: harmonic stage on
           the device, context, generate, off-diagonal and iterative kappa
  train    one step of fitting third-order force constants: linewidths and kappa forward,
           the gradient with respect to every force constant backward

listed() are the cases that are followed; draw() gives others of the same ranges. Mixed
precision is computed in 32 bits, so its results are handed out in 32 bits; the FP64 path's
in 64.
"""
from __future__ import annotations

import math
import tempfile
from pathlib import Path

import numpy as np
import torch

from tdep_gb300 import Options, Problem, QLists, ScatteringRates, synth
from tdep_gb300.autograd import linewidth_and_kappa

CELLS = {"fcc_morse": 3, "rocksalt": 6, "fluorite": 9, "l12": 12, "perovskite": 15}  # modes


def listed():
    return [
        # the smallest run there is: one atom, a coarse mesh, Gaussian smearing. Launches,
        # uploads and host work are everything; scans over many settings are made of these.
        dict(name="fcc4_fp64", op="solve", cell="fcc_morse", mesh=4, it=1, precision="fp64", isotope=True),
        # the defaults of the options (FP64, adaptive smearing, isotopes, full q' grid) on a
        # two-atom crystal with an ordinary mesh
        dict(name="rocksalt12_fp64", op="solve", cell="rocksalt", mesh=12, it=2, precision="fp64", isotope=True),
        # the largest two-atom run of the benchmark: two million q-triplets, mixed precision,
        # a 1.6 GB scattering matrix in every step of the iterative solution
        dict(name="rocksalt24_mixed", op="solve", cell="rocksalt", mesh=24, it=2, precision="mixed", isotope=False),
        # Monte-Carlo q' samples, another one for every row, on a grid that does not divide the
        # mesh; three atoms, an odd mesh
        dict(name="fluorite11_mc_mixed", op="solve", cell="fluorite", mesh=11, it=2, precision="mixed", isotope=True,
             sub=6),
        # four atoms, velocity-difference smearing, odd mesh, FP64; without isotopes, whose terms
        # between a mode at rest and itself outweigh everything else with this smearing
        dict(name="l12_9_fp64", op="solve", cell="l12", mesh=9, it=6, precision="fp64", isotope=False),
        # five atoms in FP64: the reference run against which a mixed one is checked
        dict(name="perovskite8_fp64", op="solve", cell="perovskite", mesh=8, it=2, precision="fp64", isotope=False),
        # the benchmark's default workload: five atoms, 16^3, uneven samples per q1, mixed
        dict(name="perovskite16_mixed", op="solve", cell="perovskite", mesh=16, it=2, precision="mixed", isotope=False,
             least=200, most=4000),
        # one step of a fit of the third-order force constants to a conductivity
        dict(name="train_perovskite10_mixed", op="train", cell="perovskite", mesh=10, it=2, precision="mixed",
             isotope=False),
        # three- plus four-phonon scattering, 27 x 27 pair samples per q1 (-qg4ph 3 3 3), mixed
        dict(name="fourth_perovskite8_mixed", op="solve", cell="perovskite", mesh=8, it=2, precision="mixed",
             isotope=False, pairs=27),
        # the same in FP64 on the two-atom crystal
        dict(name="fourth_rocksalt8_fp64", op="solve", cell="rocksalt", mesh=8, it=2, precision="fp64", isotope=True,
             pairs=27),
        # a disordered 40-atom supercell (120 modes, no symmetry): the large-cell path
        dict(name="supercell40_mixed", op="solve", cell="perovskite_supercell", mesh=4, it=2, precision="mixed",
             isotope=False, reps="2x2x2"),
        # everything from the files on, as the program runs it once per crystal
        dict(name="program_perovskite12_mixed", op="program", cell="perovskite", mesh=12, it=2, precision="mixed",
             isotope=True),
    ]


def draw(rng):
    """Another case of these ranges: cells of 3 to 15 modes with meshes from 4 up to what the
    listed cases take, sampled or full q' grids, both precisions, four-phonon terms, training
    steps, whole programs and supercells of 30 to 120 modes."""
    def mesh(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve", "solve", "solve", "solve", "train", "fourth", "fourth", "supercell", "program"])
    it, precision = rng.choice([1, 2, 2, 6]), rng.choice(["fp64", "mixed"])
    if kind == "supercell":
        reps, top = rng.choice([("1x1x2", 7), ("1x2x2", 5), ("2x2x2", 3)])
        return dict(op="solve", cell="perovskite_supercell", mesh=rng.randint(3, top), it=it, precision="mixed",
                    isotope=rng.random() < 0.5, reps=reps)
    cell = rng.choice(list(CELLS))
    if kind == "fourth":
        top = {"fcc_morse": 12, "rocksalt": 10, "fluorite": 9, "l12": 8, "perovskite": 8}[cell]
        return dict(op="solve", cell=cell, mesh=mesh(6, top), it=it, precision=precision, isotope=rng.random() < 0.5,
                    pairs=rng.choice([8, 18, 27]))
    if kind == "train":
        top = {"fcc_morse": 16, "rocksalt": 14, "fluorite": 12, "l12": 10, "perovskite": 10}[cell]
        if precision == "fp64":
            top -= 3
        return dict(op="train", cell=cell, mesh=mesh(4, top), it=it, precision=precision, isotope=False)
    top = {("fcc_morse", "fp64"): 20, ("rocksalt", "fp64"): 15, ("fluorite", "fp64"): 12, ("l12", "fp64"): 10,
           ("perovskite", "fp64"): 9, ("fcc_morse", "mixed"): 28, ("rocksalt", "mixed"): 22, ("fluorite", "mixed"): 18,
           ("l12", "mixed"): 15, ("perovskite", "mixed"): 13}[cell, precision]
    case = dict(op=kind, cell=cell, mesh=mesh(4, top), it=it, precision=precision, isotope=rng.random() < 0.5)
    if kind == "solve" and rng.random() < 0.3:
        case["sub"] = rng.randint(max(2, case["mesh"] // 2), case["mesh"])
    elif kind == "solve" and rng.random() < 0.3:
        case["least"], case["most"] = max(1, case["mesh"] ** 3 // 20), case["mesh"] ** 3
    return case


# ------------------------------------------------------------------------------- the calls
class State:
    """What a user's program holds between calls."""


def _reps(case):
    return tuple(int(r) for r in case["reps"].split("x"))


def _files(case, seed, tmp):
    kw = {"reps": _reps(case)} if "reps" in case else {}
    if "pairs" in case:
        kw["order4"] = True
    return synth.write_config(case["cell"], Path(tmp) / "crystal", seed=1 + seed % 9973, **kw)


def _grid(case):
    return (case["mesh"],) * 3


def _options(case, seed):
    sub = case.get("sub", -1)
    # another seed, another temperature: a run of its own
    return Options(temperature=300.0 + seed % 7, integrationtype=case["it"], sigma=1.0, seed=1 + seed % 9973,
                   precision=case["precision"], isotopescattering=case["isotope"], fourthorder="pairs" in case,
                   qg3ph=(sub,) * 3)


def _problem(case, seed):
    with tempfile.TemporaryDirectory() as tmp:
        return Problem.load(_files(case, seed, tmp), _grid(case), fourthorder="pairs" in case)


def _lists(case, seed, prob, opts):
    rng = np.random.default_rng(seed)
    pts = np.arange(1, prob.n_full + 1, dtype=np.int32)
    pick = lambda k: np.sort(rng.choice(pts, size=min(int(k), prob.n_full), replace=False))  # noqa: E731
    s3 = None
    if "least" in case:
        lo, hi = min(case["least"], prob.n_full), min(case["most"], prob.n_full)
        s3 = {q: pick(rng.integers(lo, hi + 1)) for q in range(1, prob.n_irr + 1)}
    if "pairs" in case:
        s3 = s3 or {q: pts for q in range(1, prob.n_irr + 1)}
        s4 = {q: (pick(case["pairs"]), pick(case["pairs"])) for q in range(1, prob.n_irr + 1)}
        return QLists.per_irreducible(prob, samples3=s3, samples4=s4)
    if s3 is not None:
        return QLists.per_irreducible(prob, samples3=s3)
    return QLists.monte_carlo(prob, opts)


def _kappa_bar(seed):
    a = np.random.default_rng(seed + 1).normal(size=(3, 3))
    return torch.from_numpy(np.eye(3) + 0.1 * (a + a.T))


def prepare(case, seed):
    s = State()
    s.case, s.opts = case, _options(case, seed)
    if case["op"] == "program":
        s.tmp = tempfile.TemporaryDirectory()
        s.dir = _files(case, seed, s.tmp.name)
        return s
    s.prob = _problem(case, seed)
    s.lists = _lists(case, seed, s.prob, s.opts)
    s.sr = ScatteringRates(s.prob)
    if case["op"] == "train":
        s.fc3 = torch.from_numpy(s.prob.fc3_mwm.copy())
        s.kappa_bar = _kappa_bar(seed)
    return s


def run(s):
    if s.case["op"] == "train":
        fc3 = s.fc3.clone().requires_grad_()
        lw, ks = linewidth_and_kappa(fc3, s.sr, s.opts, s.lists)
        (ks * s.kappa_bar).sum().backward()
        out = {"linewidth": lw.detach().numpy(), "kappa_sma": ks.detach().numpy(), "grad": fc3.grad.numpy()}
    elif s.case["op"] == "program":
        prob = Problem.load(s.dir, _grid(s.case), device=0)
        sr = ScatteringRates(prob)
        lw = sr.generate(s.opts)
        koff = sr.kappa_offdiag(s.opts)
        ks, ki = sr.kappa(s.opts)
        sr.close()
        out = {"linewidth": lw, "kappa_offdiag": koff, "kappa_sma": ks, "kappa_iter": ki, "Fn": sr.Fn}
    else:
        lw = s.sr.generate(s.opts, s.lists)
        ks, ki = s.sr.kappa(s.opts)
        out = {"linewidth": lw, "kappa_sma": ks, "kappa_iter": ki, "Fn": s.sr.Fn}
    if s.case["precision"] == "mixed":
        out = {k: np.asarray(v, np.float32) for k, v in out.items()}
    return out


# ------------------------------------------------------------------------------- the work
def work(case):
    """Bytes and operations of one pass, from the sizes alone. A q-triplet: the pretransform
    (N_t 27 real x complex products) and three n x n contractions of the n^3 complex tensor;
    a q-quartet likewise with n^4. The scattering matrix is written once and read once by the
    solution (which needs no more of it than that)."""
    n = CELLS.get(case["cell"]) or 15 * math.prod(_reps(case))
    full = case["mesh"] ** 3
    nsym = 1 if "reps" in case else 48
    nirr = full / 2 if nsym == 1 else (case["mesh"] + 2) ** 3 / 48 + case["mesh"]
    fc3 = {"fcc_morse": 55, "rocksalt": 158, "fluorite": 195, "l12": 220, "perovskite": 1115}.get(case["cell"], 50 * n)
    pts = case["sub"] ** 3 if "sub" in case else ((case["least"] + case["most"]) / 2 if "least" in case else full)
    triplets = nirr * min(pts, full) / 2.7
    flops = triplets * (108 * fc3 + 24 * n ** 4) * (3 if case["op"] == "train" else 1)
    xi = 8 * nirr * n * full * n
    size = 8 * full * n * (2 * n + 6) + 8 * 27 * fc3 + 2 * xi
    if "pairs" in case:
        fc4 = {"fcc_morse": 127, "rocksalt": 366, "fluorite": 455, "l12": 512, "perovskite": 2595}[case["cell"]]
        flops += nirr * case["pairs"] ** 2 / 31 * (324 * fc4 + 32 * n ** 5)
        size += 8 * 81 * fc4
    return {"bytes": int(size), "flops": int(flops + 6 * xi / 8)}


# --------------------------------------------------- the same in 64 bits, as plain torch
PI, TOL, FREQTOL, SQTOL = math.pi, 1e-5, 1e-9, 1e-10
EV = 1.0 / 27.21138602
KB, HBAR = 8.6173303e-5 * EV, 6.582119514e-16 * EV
THZ = 2 * PI * HBAR * 1e12
CHOP_V = 1e-10 / ((0.52917721067e-10 / HBAR) / 1000.0)


def _chop(k):
    return torch.where(k.abs() < k.abs().sum() * 1e-6, torch.zeros_like(k), k)


def _gauss(x, sigma):
    g = torch.exp(-0.5 * (x / sigma) ** 2) * 0.398942280401433 / sigma
    return torch.where(x.abs() > 8 * sigma, torch.zeros_like(g), g)


class Exact:
    """thermal_conductivity's scattering rates and kappa for one problem, q1 after q1."""

    def __init__(self, prob, opts, lists):
        self.p, self.o, self.lists = prob, opts, lists
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda x: torch.from_numpy(np.array(x)).to(self.dev)  # noqa: E731
        p = prob
        self.n, self.N, self.nirr = p.n_mode, p.n_full, p.n_irr
        n, N = self.n, self.N
        self.grid = [int(g) for g in p.grid]
        g0, g1, g2 = self.grid
        k = torch.arange(N, device=self.dev)
        self.xyz = torch.stack([k // (g1 * g2), (k // g2) % g1, k % g2], 1)
        self.om = t(p.omega)
        self.vel = t(p.vel)
        self.egv = torch.view_as_complex(t(p.egv))                            # [q, mode, component]
        inv = torch.where(self.om > FREQTOL, self.om.clamp(min=FREQTOL) ** -0.5, torch.zeros_like(self.om))
        self.E = (self.egv * inv[:, :, None]).transpose(1, 2).contiguous()    # [q, component, mode]
        self.full_irr = t(p.full_irr).long() - 1
        self.irr_full = t(p.irr_full).long() - 1
        self.op_cart = t(p.op_cart).reshape(-1, 3, 3).transpose(1, 2)         # row-major
        self.rl = t(p.reclat).reshape(3, 3).T / torch.tensor(self.grid, device=self.dev, dtype=torch.float64)
        self.mwm3, self.mwm4 = t(p.fc3_mwm), t(p.fc4_mwm)
        self.images = self._images(p)
        om, T = self.om[self.irr_full], opts.temperature
        live = om >= FREQTOL
        x = om.clamp(min=FREQTOL) / (KB * T)
        be = torch.where(x > 100, torch.zeros_like(x), 1 / (torch.exp(x) - 1))
        be = be if not opts.classical else KB * T / om.clamp(min=FREQTOL)
        self.be = torch.where(live, be, torch.zeros_like(be))
        sq = ((self.vel[self.irr_full].abs() @ self.rl) ** 2 * 0.5).amax(-1)
        sq = torch.where(live, sq, torch.zeros_like(sq))
        self.weight = t(p.irr_weight)
        self.thresh = float((sq * self.weight[:, None]).sum(0).max()) * 1e-4
        self.sigsq = sq + self.thresh
        self.sigma = opts.sigma * THZ
        cv = KB * x * x * torch.exp(x) / (torch.exp(x) - 1) ** 2
        cv = torch.where(x > 21, KB * x * x * torch.exp(-x), torch.where(x < 2e-2, KB * (1 - x ** 2 / 12 + x ** 4 / 240), cv))
        self.cv = torch.where(live & (x <= 200), cv, torch.zeros_like(cv))
        rows = {}
        for r, (q1, b1) in enumerate(zip(lists.row_q1, lists.row_b1)):
            rows.setdefault(int(q1) - 1, []).append((r, int(b1) - 1))
        self.rows = rows
        d, dm = t(p.degen).long(), t(p.degen_mode).long() - 1
        f = self.irr_full
        first = torch.arange(n, device=self.dev) < d[f][:, :, None]
        self.mean = torch.zeros(self.nirr, n, n, device=self.dev, dtype=torch.float64)  # degenerate average
        self.mean.scatter_add_(2, dm[f].clamp(min=0), first / d[f][:, :, None].double())

    def _images(self, p):
        """Images of every mesh point under the operations of each little group (-1 off the mesh)."""
        out = []
        L = math.lcm(*self.grid)
        mul = torch.tensor([L // g for g in self.grid], device=self.dev)
        for i in range(self.nirr):
            ops = np.abs(p.irr_ops[i][: p.irr_nop[i]]) - 1
            R = torch.from_numpy(p.op_recfrac[ops].reshape(-1, 3, 3).transpose(0, 2, 1).astype(np.int64)).to(self.dev)
            w = (R.double() @ (self.xyz * mul).double().T).round().long() % L   # [op, 3, point]
            on = (w % mul[None, :, None] == 0).all(1)
            g = w // mul[None, :, None]
            out.append(torch.where(on, (g[:, 0] * self.grid[1] + g[:, 1]) * self.grid[2] + g[:, 2], -1))
        return out

    def _minus(self, *qs):
        s = -sum(self.xyz[q] for q in qs)
        s = s % torch.tensor(self.grid, device=self.dev)
        return (s[:, 0] * self.grid[1] + s[:, 1]) * self.grid[2] + s[:, 2]

    def _counts(self, q1, ptr, *lists):
        """How often each row of q1 samples a point (or a pair): (keys, [mode, key] counts)."""
        per, keys = [], []
        for r, b1 in self.rows[q1]:
            a = [x[ptr[r]:ptr[r + 1]].astype(np.int64) - 1 for x in lists]
            key = a[0] if len(a) == 1 else (a[0][:, None] * self.N + a[1][None, :]).ravel()
            u, c = np.unique(key, return_counts=True)
            keys.append(u)
            per.append((b1, u, c / len(a[0]) ** len(a)))
        every = np.unique(np.concatenate(keys))
        w = np.zeros((self.n, every.size))
        for b1, u, c in per:
            w[b1, np.searchsorted(every, u)] = c
        return torch.from_numpy(every).to(self.dev), torch.from_numpy(w).to(self.dev)

    def _ptf(self, mwm, atoms, lv, qs, m):
        """Force constants summed with their phases: [item, n, ..., n]."""
        n, K = self.n, 3 ** m
        a = torch.from_numpy(np.array(atoms)).long().to(self.dev) - 1
        l = torch.from_numpy(np.array(lv)).to(self.dev).double().reshape(-1, m - 1, 3)
        frac = self.xyz.double() / torch.tensor(self.grid, device=self.dev)
        arg = sum(frac[q] @ l[:, i].T for i, q in enumerate(qs))
        ph = torch.polar(torch.ones_like(arg), -2 * PI * (arg - arg.round()))
        e = torch.arange(K, device=self.dev)
        idx = torch.zeros(a.shape[0], K, dtype=torch.long, device=self.dev)
        for d in range(m):  # first index fastest inside a force constant, slowest in the tensor
            idx = idx * n + 3 * a[:, d: d + 1] + (e // 3 ** d) % 3
        out = torch.zeros(len(qs[0]), n ** m, dtype=torch.complex128, device=self.dev)
        return out.index_add(1, idx.ravel(), (ph[:, :, None] * mwm[None]).reshape(len(qs[0]), -1)).reshape(-1, *[n] * m)

    def _width(self, q1, qs):
        """Smearing of all mode combinations of [q1, q2, ...]: broadcastable [item, n, ...]."""
        m = len(qs) + 1
        shape = lambda x, d: x.reshape(*x.shape[:1], *[self.n if k == d else 1 for k in range(m)])  # noqa: E731
        if self.o.integrationtype == 1:
            return torch.full((1,) * (m + 1), self.sigma, dtype=torch.float64, device=self.dev)
        if self.o.integrationtype == 2:
            s = [self.sigsq[q1][None]] + [self.sigsq[self.full_irr[q]] for q in qs]
            return torch.sqrt(sum(shape(x, d) for d, x in enumerate(s)))
        v = [self.vel[self.irr_full[q1]][None]] + [self.vel[q] for q in qs]
        total, pairs = self.thresh, m * (m - 1) // 2
        for i in range(m):
            for j in range(i + 1, m):
                d = ((v[i][:, :, None, :] - v[j][:, None, :, :]) @ self.rl) ** 2
                d = torch.sqrt(0.5 * d.amax(-1)) / pairs
                total = total + d.reshape(d.shape[0], *[self.n if k in (i, j) else 1 for k in range(m)])
        return total

    def _equivalent(self, imgs, own):
        """The distinct images of each item: (images [op, item] per point, included [op, item])."""
        on = torch.stack([x >= 0 for x in imgs]).all(0)
        srt = torch.stack([torch.where(on, x, o[None]) for x, o in zip(imgs, own)]).sort(0).values
        key = srt[0]
        for x in srt[1:]:
            key = key * self.N + x
        if len(own) == 3:
            key = torch.where(on, key, -1)
        imgs = [torch.where(on, x, o[None]) for x, o in zip(imgs, own)]
        inc = torch.ones_like(on)
        for j in range(key.shape[0] - 1):
            inc[j] = ~(key[j + 1:] == key[j]).any(0)
        return imgs, inc

    def third(self, q1, mwm):
        """(gamma [mode], od [mode, point, mode] before symmetrisation) of q1's three-phonon terms."""
        n, f1, im = self.n, int(self.irr_full[q1]), self.images[q1]
        q2, w = self._counts(q1, self.lists.ptr3, self.lists.list3)
        q3 = self._minus(torch.full_like(q2, f1), q2)
        x, y = im[:, q2], im[:, q3]
        bad = ((torch.minimum(x, y) > q2[None]) & (x >= 0) & (y >= 0)).any(0) | (q3 < q2)
        q2, q3, w = q2[~bad], q3[~bad], w[:, ~bad]
        gamma = torch.zeros(n, dtype=torch.float64, device=self.dev)
        od = torch.zeros(n, self.N, n, dtype=torch.float64, device=self.dev)
        step = max(1, int(3e9 / (16 * (4 * n ** 3 + 54 * self.p.n_fc3))))
        for i in range(0, len(q2), step):
            gamma = gamma + self._third(q1, q2[i:i + step], q3[i:i + step], w[:, i:i + step], mwm, od)
        return gamma, od

    def _third(self, q1, q2, q3, w, mwm, od):
        f1, im = int(self.irr_full[q1]), self.images[q1]
        (x, y), inc = self._equivalent([im[:, q2], im[:, q3]], [q2, q3])
        P = self._ptf(mwm, self.p.fc3_atoms, self.p.fc3_lv, [q2, q3], 3)
        P = torch.einsum("tabc,ax->txbc", P, self.E[f1])
        P = torch.einsum("txbc,tby->txyc", P, self.E[q2])
        P = torch.einsum("txyc,tcz->txyz", P, self.E[q3])
        psi = (P.real ** 2 + P.imag ** 2) * (PI / 16)
        o1, o2, o3 = self.om[f1][None, :, None, None], self.om[q2][:, None, :, None], self.om[q3][:, None, None, :]
        sg = self._width(q1, [q2, q3])
        d0 = _gauss(o1 + o2 - o3, sg) - _gauss(o1 - o2 + o3, sg)
        d1 = _gauss(o1 - o2 - o3, sg) - _gauss(o1 + o2 + o3, sg)
        n2, n3 = self.be[self.full_irr[q2]][:, None, :, None], self.be[self.full_irr[q3]][:, None, None, :]
        skip = (o1 < FREQTOL) | (o2 < FREQTOL) | (o3 < FREQTOL) | ((o1 - o2).abs() < FREQTOL)
        skip = skip | ((o1 - o3).abs() < FREQTOL) | ((o2 - o3).abs() < FREQTOL)
        wt = w.T * torch.where(q2 == q3, 1.0, 2.0)[:, None]
        F = psi * ((n2 - n3) * d0 + (n2 + n3 + 1) * d1) * wt[:, :, None, None]
        F = torch.where(skip, torch.zeros_like(F), F)
        gamma = (F.sum((2, 3)) * inc.sum(0)[:, None]).sum(0)
        if not mwm.requires_grad:
            self._scatter(od, F, inc, [x, y], [o2, o3], o1)
        return gamma

    def _scatter(self, od, F, inc, imgs, oms, o1):
        _, item = inc.nonzero(as_tuple=True)
        m = len(imgs) + 1
        for d, (x, o) in enumerate(zip(imgs, oms)):
            v = 2 * F * o / o1.clamp(min=FREQTOL)
            others = [k for k in range(2, m + 1) if k != d + 2]
            od.index_add_(1, x[inc], v.sum(others)[item].transpose(0, 1).contiguous())

    def fourth(self, q1):
        n, f1, im = self.n, int(self.irr_full[q1]), self.images[q1]
        key, w = self._counts(q1, self.lists.ptr4, self.lists.list4a, self.lists.list4b)
        q2, q3 = key // self.N, key % self.N
        q4 = self._minus(torch.full_like(q2, f1), q2, q3)
        ok = (q3 >= q2) & (q4 >= q3)
        q2, q3, q4, w = q2[ok], q3[ok], q4[ok], w[:, ok]
        on = (im[:, q2] >= 0) & (im[:, q3] >= 0) & (im[:, q4] >= 0)
        s = torch.stack([im[:, q2], im[:, q3], im[:, q4]]).sort(0).values
        ok = ~(((s[0] > q2) | (s[1] > q3)) & on).any(0)
        q2, q3, q4, w = q2[ok], q3[ok], q4[ok], w[:, ok]
        gamma = torch.zeros(n, dtype=torch.float64, device=self.dev)
        od = torch.zeros(n, self.N, n, dtype=torch.float64, device=self.dev)
        step = max(1, int(4e9 / (16 * (6 * n ** 4 + 162 * self.p.n_fc4))))
        for i in range(0, len(q2), step):
            gamma = gamma + self._fourth(q1, q2[i:i + step], q3[i:i + step], q4[i:i + step], w[:, i:i + step], od)
        return gamma, od

    def _fourth(self, q1, q2, q3, q4, w, od):
        f1, im = int(self.irr_full[q1]), self.images[q1]
        imgs, inc = self._equivalent([im[:, q2], im[:, q3], im[:, q4]], [q2, q3, q4])
        P = self._ptf(self.mwm4, self.p.fc4_atoms, self.p.fc4_lv, [q2, q3, q4], 4)
        P = torch.einsum("tabcd,ax->txbcd", P, self.E[f1])
        P = torch.einsum("txbcd,tby->txycd", P, self.E[q2])
        P = torch.einsum("txycd,tcz->txyzd", P, self.E[q3])
        P = torch.einsum("txyzd,tdw->txyzw", P, self.E[q4])
        psi = (P.real ** 2 + P.imag ** 2) * (PI / 96)
        del P
        shape = lambda x, d: x.reshape(x.shape[0], *[self.n if k == d else 1 for k in range(4)])  # noqa: E731
        om = [shape(x, d) for d, x in enumerate([self.om[f1][None], self.om[q2], self.om[q3], self.om[q4]])]
        o1, o2, o3, o4 = om
        a, b, c = (shape(self.be[self.full_irr[q]], d) for d, q in ((1, q2), (2, q3), (3, q4)))
        sg = self._width(q1, [q2, q3, q4])
        mult = torch.where((q2 == q3) & (q3 == q4), 1.0, torch.where((q2 == q3) | (q3 == q4) | (q2 == q4), 3.0, 6.0))
        other = torch.where(mult == 6.0, 2.0, 1.0)
        mult, other = mult.reshape(-1, 1, 1, 1, 1), other.reshape(-1, 1, 1, 1, 1)
        a1, b1, c1 = a + 1, b + 1, c + 1
        F = mult * (a1 * b1 * c1 - a * b * c) * (_gauss(o1 - o2 - o3 - o4, sg) - _gauss(o1 + o2 + o3 + o4, sg))
        F = F + other * (3 * a * b1 * c1 - a1 * b * c) * (_gauss(o1 + o2 - o3 - o4, sg) - _gauss(o1 - o2 + o3 + o4, sg))
        F = F + other * (3 * b * a1 * c1 - b1 * a * c) * (_gauss(o1 - o2 + o3 - o4, sg) - _gauss(o1 + o2 - o3 + o4, sg))
        F = F + other * (3 * c * b1 * a1 - c1 * b * a) * (_gauss(o1 - o2 - o3 + o4, sg) - _gauss(o1 + o2 + o3 - o4, sg))
        F = F * psi * w.T.reshape(-1, self.n, 1, 1, 1)
        F = torch.where((o1 < FREQTOL) | (o2 < FREQTOL) | (o3 < FREQTOL) | (o4 < FREQTOL), torch.zeros_like(F), F)
        self._scatter(od, F, inc, imgs, [o2, o3, o4], o1)
        return (F.sum((2, 3, 4)) * inc.sum(0)[:, None]).sum(0)

    def isotope(self, q1):
        f1 = int(self.irr_full[q1])
        o1, o2 = self.om[f1][:, None, None], self.om[None]
        amp = (self.egv[f1].conj()[:, None, None] * self.egv[None]).abs()
        amp = amp.reshape(*amp.shape[:3], -1, 3).sum(-1) ** 2 @ torch.from_numpy(self.p.mass_disorder.copy()).to(self.dev)
        if self.o.integrationtype == 1:
            sg = torch.full_like(o2, self.sigma)
        elif self.o.integrationtype == 2:
            sg = torch.sqrt(self.sigsq[q1][:, None, None] + self.sigsq[self.full_irr][None])
        else:
            sg = torch.sqrt(0.5 * ((self.vel @ self.rl) ** 2).amax(-1))[None] + self.thresh
        f = amp * (PI / 4 / self.N) * o1 * o2 * _gauss(o1 - o2, sg)
        f = torch.where((o1 < FREQTOL) | (o2 < FREQTOL), torch.zeros_like(f), f)
        return f.sum((1, 2)), f * o2 / o1.clamp(min=FREQTOL)

    def distribute(self, q1, od, ptr, lst):
        """Averages of the positive terms over the orbits whose first point a row has sampled."""
        im = self.images[q1]
        first = torch.where(im >= 0, im, self.N).amin(0) == torch.arange(self.N, device=self.dev)
        rep = first.nonzero().ravel()
        im = im[:, rep]
        on = (im >= 0)[None, :, :, None]
        seen = torch.zeros(self.n, self.N, dtype=torch.bool, device=self.dev)
        for r, b1 in self.rows[q1]:
            seen[b1, torch.from_numpy(lst[ptr[r]:ptr[r + 1]].astype(np.int64) - 1).to(self.dev)] = True
        for b1 in range(self.n):  # a mode at a time: the images of a whole orbit at once
            v = od[b1][im.clamp(min=0)]
            pos = (v > 0) & on[0]
            nn = pos.sum(0)
            mean = torch.where(pos, v, torch.zeros_like(v)).sum(0) / nn.clamp(min=1)
            put = (nn > 0) & seen[b1, rep][:, None]
            for j in range(im.shape[0]):
                p = torch.where(im[j] >= 0, im[j], rep)
                od[b1, p] = torch.where(put & on[0, j], mean, od[b1, p])
        return od

    def symmetrise(self, q1, xi):
        im = self.images[q1]
        on = (im >= 0).double()
        # the mean over a point's images is the same for all points of an orbit
        out = torch.zeros_like(xi)
        for j in range(im.shape[0]):
            out += xi[:, im[j].clamp(min=0)] * on[j][None, :, None]
        return out / on.sum(0)[None, :, None].clamp(min=1)

    def scattering(self, matrix=True):
        """Linewidths [n_irr, mode] after the degenerate average; self.xi when matrix."""
        gamma = torch.zeros(self.nirr, self.n, dtype=torch.float64, device=self.dev)
        xi = []
        for q1 in sorted(self.rows):
            g, od = self.third(q1, self.mwm3)
            od = self.distribute(q1, od, self.lists.ptr3, self.lists.list3) if matrix else od
            if self.o.isotopescattering:
                gi, oi = self.isotope(q1)
                g, od = g + gi, od + oi
            if self.o.fourthorder:
                g4, o4 = self.fourth(q1)
                g, od = g + g4, od + self.distribute(q1, o4, self.lists.ptr4, self.lists.list4a)
            gamma[q1] = g
            if matrix:
                b1 = torch.tensor([b for _, b in self.rows[q1]], device=self.dev)
                xi.append(self.symmetrise(q1, od)[b1].reshape(len(b1), -1))
        self.xi = torch.cat(xi) if matrix else None
        self.live = self.om[self.irr_full] >= FREQTOL
        return torch.where(self.live, (self.mean @ gamma[:, :, None])[..., 0], torch.zeros_like(gamma))

    def kappa_of(self, F):
        v = self.vel[self.irr_full]
        k = (F[:, :, :, None] * v[:, :, None, :] * (self.cv * self.weight[:, None])[:, :, None, None]).sum((0, 1))
        return _chop(torch.einsum("oik,kl,ojl->ij", self.op_cart, k, self.op_cart) / len(self.op_cart) / self.p.volume)

    def symmetric(self, k):
        return _chop(torch.einsum("oik,kl,ojl->ij", self.op_cart, k, self.op_cart) / len(self.op_cart))

    def start(self, lw):
        ok = lw > FREQTOL
        return torch.where(ok[:, :, None], self.vel[self.irr_full] / (2 * torch.where(ok, lw, torch.ones_like(lw)))[:, :, None],
                           torch.zeros_like(lw)[:, :, None])

    def solve(self, lw, tol, maxiter):
        F0, qs = self.start(lw), 2 * lw
        F, mixing, seen = F0.clone(), 0.95, []
        op = torch.from_numpy(np.array(self.p.full_op)).long().to(self.dev)
        m = self.op_cart[op.abs() - 1] * torch.sign(op).double()[:, None, None]
        row = torch.cat([torch.tensor([[q1, b] for _, b in self.rows[q1]], device=self.dev) for q1 in sorted(self.rows)])
        for it in range(1, maxiter + 1):
            full = torch.einsum("qij,qbj->qbi", m, F[self.full_irr]).reshape(-1, 3)
            prod = torch.zeros_like(F)
            prod[row[:, 0], row[:, 1]] = self.xi @ full
            new = torch.where((qs < FREQTOL)[:, :, None], torch.zeros_like(F), -prod / qs.clamp(min=FREQTOL)[:, :, None])
            for b in range(self.n):  # in place, mode after mode, F0 added as it goes
                w = self.mean[:, b]
                mean = torch.einsum("qk,qkd->qd", w, new)
                new = torch.where((w > 0)[:, :, None], mean[:, None], new)
                new[:, b] = new[:, b] + F0[:, b]
            change, size = ((F - new) ** 2).sum(-1), (F ** 2).sum(-1)
            seen.append(float(torch.where(size > SQTOL, change / size.clamp(min=SQTOL), torch.zeros_like(size)).sum())
                        / self.nirr / self.n)
            F = F * (1 - mixing) + mixing * new
            if it >= 3 and sum(seen[-3:]) < tol:
                break
            if it > 15 and mixing > 0.5:
                mixing *= 0.98
        return F

    def offdiag(self, lw):
        """Coherence term: velocity matrix averaged over the little group, then over the star."""
        p, n, na = self.p, self.n, self.p.n_atom
        t = lambda x: torch.from_numpy(np.array(x)).to(self.dev)  # noqa: E731
        D = torch.view_as_complex(t(p.irr_dyngrad)).transpose(2, 3)  # [q, xyz, row, column]
        q_full, shift, fmap = t(p.q_full), t(p.atom_shift), t(p.op_fmap).long() - 1
        out = torch.zeros(3, 3, dtype=torch.float64, device=self.dev)
        star = t(p.full_op).long().abs() - 1
        for i in range(self.nirr):
            f, v = int(self.irr_full[i]), 0
            om = self.om[f]
            s = torch.where(om > FREQTOL, (2 * om.clamp(min=FREQTOL)) ** -0.5, torch.zeros_like(om))
            ops = [int(x) for x in p.irr_ops[i][: p.irr_nop[i]]]
            for op in ops:
                o = abs(op) - 1
                ph = -2 * PI * (shift[o] @ q_full[f])
                G = torch.zeros(na, 3, na, 3, dtype=torch.complex128, device=self.dev)
                G[fmap[o], :, torch.arange(na, device=self.dev), :] = (
                    torch.polar(torch.ones_like(ph), ph)[:, None, None] * self.op_cart[o][None])
                e = G.reshape(n, n) @ self.egv[f].T
                e = (e.conj() if op < 0 else e) * s[None]
                v = v + e.conj().T @ D[i] @ e
            v = (v / len(ops)).real
            v = torch.where(v.abs() < CHOP_V, torch.zeros_like(v), v)
            m = self.op_cart[star[self.full_irr == i]]
            vv = torch.einsum("sak,kij,sbl,lij->ijab", m, v, m, v) / len(m)
            o, g, c = om, lw[i], self.cv[i] if not self.o.classical else torch.full_like(om, KB)
            ok = (o >= FREQTOL) & (g >= FREQTOL)
            gg = g[:, None] + g[None]
            tau = gg / (gg ** 2 + (o[:, None] - o[None]) ** 2) * 0.5 * (c[:, None] + c[None])
            tau = torch.where(ok[:, None] & ok[None] & ~torch.eye(n, dtype=torch.bool, device=self.dev), tau, torch.zeros_like(tau))
            out += (vv * tau[:, :, None, None]).sum((0, 1)) * self.weight[i] / p.volume
        return self.symmetric(_chop(out))

    def gradient(self, lw, kappa_bar):
        """d (kappa_bar : kappa_sma) / d force constants, by reverse mode through the above."""
        g = lw.clone().requires_grad_()
        (self.symmetric(self.kappa_of(self.start(g))) * kappa_bar).sum().backward()
        lam = (self.mean.transpose(1, 2) @ torch.where(self.live, g.grad, torch.zeros_like(lw))[:, :, None])[..., 0]
        mwm = self.mwm3.clone().requires_grad_()
        for q1 in sorted(self.rows):
            n, f1, im = self.n, int(self.irr_full[q1]), self.images[q1]
            q2, w = self._counts(q1, self.lists.ptr3, self.lists.list3)
            q3 = self._minus(torch.full_like(q2, f1), q2)
            x, y = im[:, q2], im[:, q3]
            bad = ((torch.minimum(x, y) > q2[None]) & (x >= 0) & (y >= 0)).any(0) | (q3 < q2)
            q2, q3, w = q2[~bad], q3[~bad], w[:, ~bad]
            step = max(1, int(2e9 / (16 * (12 * n ** 3 + 108 * self.p.n_fc3))))
            for i in range(0, len(q2), step):
                (self._third(q1, q2[i:i + step], q3[i:i + step], w[:, i:i + step], mwm, None) * lam[q1]).sum().backward()
        return mwm.grad


def exact(case, seed):
    if not torch.cuda.is_available():
        return None
    prob, opts = _problem(case, seed), _options(case, seed)
    lists = QLists.monte_carlo(prob, opts) if case["op"] == "program" else _lists(case, seed, prob, opts)
    x = Exact(prob, opts, lists)
    lw = x.scattering(matrix=case["op"] != "train")
    out = {"linewidth": lw, "kappa_sma": x.symmetric(x.kappa_of(x.start(lw)))}
    if case["op"] == "train":
        out["grad"] = x.gradient(lw, _kappa_bar(seed).to(x.dev))
        return {k: out[k].cpu().numpy() for k in ("linewidth", "kappa_sma", "grad")}
    F = x.solve(lw, opts.itertol, opts.itermaxsteps)
    out["kappa_iter"], out["Fn"] = x.symmetric(x.kappa_of(F)), F
    order = ["linewidth", "kappa_sma", "kappa_iter", "Fn"]
    if case["op"] == "program":
        out["kappa_offdiag"] = x.offdiag(lw)
        order.insert(1, "kappa_offdiag")
    return {k: out[k].cpu().numpy() for k in order}
