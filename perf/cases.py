"""What the speed of this engine is measured on: the calls its users make.

Kinds of case
  curve     run_curve: a whole n(mu) curve of a small lattice, every sector and
            momentum block (a twist average calls it once per twist)
  block     one momentum block as the curve loop visits it: sector tables,
            FTLM spectrum, Boltzmann sums, read back (the unit of a big lattice)
  spectrum  sector tables and one block's Ritz values and weights, few vectors
            and few steps (training spectra of the twist surrogate)
  apply     H*V of a momentum block on host vectors
  train     the surrogate network: created, trained, its weights read back

Every model takes its twist from the seed, and the random vectors theirs.
Results of mixed-precision runs (FP32 vectors) are given in single precision,
which is what they hold; FP64 runs give doubles.
"""
import math
import random

import numpy as np
import torch

import ftlm_extended_hubbard_development_b200 as pkg
from ftlm_extended_hubbard_development_b200 import engine as E

L2_BYTES = 126 << 20
MU = {"mu_min": -3.0, "mu_max": 4.0, "mu_points": 141}


def _curve(name, lx, ly, **kw):
    c = {**({"name": name} if name else {}), "kind": "curve", "lx": lx, "ly": ly, "tp": 0.0, "u": 8.0, "v": 0.0, "betas": "5.0", **MU,
         "samples": 5, "steps": 80, "threshold": 256, "precision": "fp64", "start": "gaussian", "ed": False}
    c.update(kw)
    return c


def _block(name, lx, ly, nup, ndn, mx, my, **kw):
    c = {**({"name": name} if name else {}), "kind": "block", "lx": lx, "ly": ly, "tp": 0.0, "u": 7.0, "v": 0.0, "nup": nup, "ndn": ndn,
         "mx": mx, "my": my, "betas": "2.857142857142857,12.5", **MU, "samples": 128, "steps": 80,
         "precision": "mixed", "start": "philox"}
    c.update(kw)
    return c


def listed():
    return [
        # H*V of a tiny block, one vector: call latency, nothing else
        {"name": "apply_3x2", "kind": "apply", "lx": 3, "ly": 2, "tp": 0.2, "u": 8.0, "v": 1.5, "nup": 3, "ndn": 3,
         "mx": 1, "my": 0, "nvec": 1, "precision": "fp64"},
        # H*V of an ordinary block on 16 host vectors, as an outside solver calls it
        {"name": "apply_4x4_34", "kind": "apply", "lx": 4, "ly": 4, "tp": -0.25, "u": 7.0, "v": 1.0, "nup": 3,
         "ndn": 4, "mx": 1, "my": 0, "nvec": 16, "precision": "mixed"},
        # the smallest lattice with the default run (5 vectors, 40 steps): every block is exact
        _curve("curve_2x2", 2, 2, tp=0.2, u=4.0, v=1.0, betas="1.5", mu_min=-2.0, mu_max=6.0, mu_points=33, steps=40),
        # the FTLM-against-ED check lattice in production settings
        _curve("curve_4x2_mixed", 4, 2, betas="20.0", mu_min=-5.0, mu_max=15.0, mu_points=81, samples=32, steps=120,
               precision="mixed", start="philox"),
        # its exact counterpart: every block diagonalised
        _curve("curve_4x2_ed", 4, 2, betas="20.0", mu_min=-5.0, mu_max=15.0, mu_points=81, ed=True),
        # an odd lattice with all couplings on, default vectors and steps, two temperatures
        _curve("curve_3x3_fp64", 3, 3, tp=0.2, u=8.0, v=1.5, betas="2.5,10.0"),
        # a mid-size block at the default settings of the executable: 5 FP64 vectors
        _block("block_4x4_44_fp64", 4, 4, 4, 4, 1, 2, tp=-0.25, v=1.0, samples=5, precision="fp64", start="gaussian"),
        # production curve: a sector of ordinary size, all vectors in one sweep
        _block("block_4x4_55", 4, 4, 5, 5, 0, 0, mu_points=281),
        # production curve: its largest sector
        _block("block_4x4_88", 4, 4, 8, 8, 0, 0, samples=64, steps=40, mu_points=281),
        # 18 sites, all couplings on, 16 vectors: long rows, narrow sweeps
        _block("block_6x3_55", 6, 3, 5, 5, 2, 1, tp=0.2, u=8.0, v=1.5, betas="10.0", mu_min=-4.0, mu_max=8.0,
               mu_points=121, samples=16, steps=100),
        # surrogate training data: 2 vectors x 20 steps on a large block
        {"name": "spectrum_4x4_66", "kind": "spectrum", "lx": 4, "ly": 4, "tp": -0.25, "u": 7.0, "v": 1.0, "nup": 6,
         "ndn": 6, "mx": 1, "my": 0, "samples": 2, "steps": 20, "precision": "mixed", "start": "philox"},
        # surrogate training: 36 twists x 620 blocks of a 4x2 lattice, mini-batches of 512
        {"name": "train_4x2", "kind": "train", "rows": 22320, "n_in": 32, "width": 128, "depth": 3, "n_out": 32,
         "epochs": 2, "batch": 512, "lr": 1e-3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rows(c):
    """Rows of one momentum block, nearly."""
    n = c["lx"] * c["ly"]
    return math.comb(n, c["nup"]) * math.comb(n, c["ndn"]) / n


def _hops(c):
    """Mean hops out of a row of a (nup, ndn) block."""
    n = c["lx"] * c["ly"]
    ndir = 8 if c["tp"] else 4
    return ndir * (c["nup"] * (n - c["nup"]) + c["ndn"] * (n - c["ndn"])) / max(n - 1, 1)


def _couplings(rng):
    return {"tp": rng.choice([0.0, 0.0, 0.2, -0.25]), "u": rng.choice([4.0, 7.0, 8.0]), "v": rng.choice([0.0, 1.0, 1.5])}


def _sector(rng, lattices, lo, hi):
    while True:
        lx, ly = rng.choice(lattices)
        n = lx * ly
        c = {"lx": lx, "ly": ly, "nup": rng.randint(1, n - 1), "ndn": rng.randint(1, n - 1), "mx": rng.randrange(lx),
             "my": rng.randrange(ly), **_couplings(rng)}
        if lo <= _rows(c) <= hi:
            return c


def draw(rng):
    kind = rng.choice(["apply", "curve", "curve", "ed", "block", "block", "block", "spectrum", "train"])
    precision = rng.choice(["mixed", "fp64"])
    start = rng.choice(["philox", "gaussian"])
    if kind == "apply":
        c = _sector(rng, [(3, 2), (4, 2), (3, 3), (4, 3), (4, 4), (6, 3)], 20, 7e4)
        return {"kind": "apply", **c, "nvec": _log(rng, 1, 24), "precision": precision}
    if kind in ("curve", "ed"):
        lx, ly = rng.choice([(2, 2), (3, 2), (6, 1), (4, 2), (8, 1)] + ([] if kind == "ed" else [(3, 3)]))
        return _curve("", lx, ly, **_couplings(rng), betas=rng.choice(["1.5", "5.0", "20.0", "2.5,10.0"]),
                      mu_points=rng.randint(21, 201), samples=_log(rng, 2, 32), steps=_log(rng, 20, 120),
                      threshold=_log(rng, 32, 256), precision=precision, start=start, ed=kind == "ed")
    if kind == "block":
        while True:
            c = _sector(rng, [(4, 3), (5, 3), (4, 4), (4, 4), (6, 3)], 3e3, 6e6)
            c |= {"samples": _log(rng, 1, 128), "steps": _log(rng, 20, 100)}
            if start == "gaussian" and c["samples"] * _rows(c) > 4e6:
                continue
            if _rows(c) * (_hops(c) + 12) * c["samples"] * c["steps"] <= (5e11 if precision == "mixed" else 2e11):
                break
        return {**_block("", 0, 0, 0, 0, 0, 0), **c, "precision": precision, "start": start,
                "mu_points": rng.randint(33, 281)}
    if kind == "spectrum":
        c = _sector(rng, [(4, 4), (4, 4), (5, 3), (6, 3)], 5e4, 5e6)
        return {"kind": "spectrum", **c, "samples": rng.randint(1, 4), "steps": rng.randint(10, 24),
                "precision": "mixed", "start": "philox"}
    return {"kind": "train", "rows": _log(rng, 2000, 22000), "n_in": rng.randint(20, 52), "width": 128, "depth": 3,
            "n_out": 32, "epochs": 1, "batch": rng.choice([128, 256, 500, 512]), "lr": 1e-3}


# ------------------------------------------------------------------ the calls


def _model(case, seed):
    r = random.Random(seed)
    return pkg.Model(lx=case["lx"], ly=case["ly"], tp=case["tp"], u=case["u"], v=case["v"], phix=r.random(),
                     phiy=r.random())


def _opts(case, seed):
    return pkg.RunOpts(samples=case.get("samples", 5), lanczos_steps=case.get("steps", 80),
                       exact_block_threshold=case.get("threshold", 256), seed=12345 + seed,
                       precision=E.PREC_MIXED if case["precision"] == "mixed" else E.PREC_FP64,
                       start_vector=E.START_PHILOX_PHASE if case.get("start") == "philox" else E.START_REF_GAUSSIAN)


def _grid(case):
    betas = [float(b) for b in case["betas"].split(",")]
    return betas, pkg.linspace(case["mu_min"], case["mu_max"], case["mu_points"])


def _vectors(case, seed):
    g = np.random.default_rng(seed)
    shape = (_dim(case), case["nvec"])
    return g.standard_normal(shape) + 1j * g.standard_normal(shape)


def _dim(case):
    """Dimension of block (mx, my): (1/N) sum over translations of the character."""
    lx, ly = case["lx"], case["ly"]
    n = lx * ly
    tot = 0.0
    for s in range(n):
        perm = [((q // lx + s // lx) % ly) * lx + (q % lx + s % lx) % lx for q in range(n)]
        tr = _trace(perm, case["nup"]) * _trace(perm, case["ndn"])
        tot += tr * math.cos(2 * math.pi * (case["mx"] * (s % lx) / lx + case["my"] * (s // lx) / ly))
    return round(tot / n)


def _trace(perm, k):
    """Trace of a site permutation on k fermions: coefficient of x^k in prod over cycles (1 - (-x)^len)."""
    poly, seen = [1] + [0] * k, set()
    for s in range(len(perm)):
        length = 0
        while s not in seen:
            seen.add(s)
            s = perm[s]
            length += 1
        if length:
            sign = 1 if length % 2 else -1
            poly = [poly[i] + (sign * poly[i - length] if i >= length else 0) for i in range(k + 1)]
    return poly[k]


def _train_data(case, seed):
    """Rows as the surrogate makes them: sin/cos of two twist phases and harmonics, one-hot quantum
    numbers, standardised targets, positive level importances as the mask."""
    g = np.random.default_rng(seed)
    n, nf = case["rows"], case["n_in"]
    x = np.zeros((n, nf), np.float32)
    ph = g.uniform(0, math.pi, (n, 2))
    for h in (1, 2):
        for a in (0, 1):
            x[:, 4 * (h - 1) + 2 * a] = np.sin(h * ph[:, a])
            x[:, 4 * (h - 1) + 2 * a + 1] = np.cos(h * ph[:, a])
    hot = np.array_split(np.arange(8, nf), 4)
    for cols in hot:
        x[np.arange(n), g.choice(cols, n)] = 1.0
    mix = g.standard_normal((nf, case["n_out"])) / math.sqrt(nf)
    t = (np.sin(x @ mix) + 0.1 * g.standard_normal((n, case["n_out"]))).astype(np.float32)
    m = (1e-3 + g.random((n, case["n_out"])) ** 4).astype(np.float32)
    return x, t, m


def _init_params(case, seed):
    g = np.random.default_rng(seed + 1)
    sizes = [case["n_in"]] + [case["width"]] * case["depth"] + [case["n_out"]]
    p = []
    for fi, fo in zip(sizes, sizes[1:]):
        a = math.sqrt(6.0 / (fi + fo))
        p += [g.uniform(-a, a, fi * fo), np.zeros(fo)]
    return np.concatenate(p).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "seed": seed}
    if kind == "train":
        state["data"] = _train_data(case, seed)
        state["p0"] = _init_params(case, seed)
        return state
    state["model"], state["opts"] = _model(case, seed), _opts(case, seed)
    if kind in ("curve", "block"):
        state["grid"] = _grid(case)
    if kind == "curve":
        return state
    state["engine"] = pkg.Engine(state["model"], state["opts"])
    if kind == "apply":
        state["engine"].sector_prepare(case["nup"], case["ndn"])
        state["x"] = _vectors(case, seed)
    return state


def _as_held(case, a):
    return np.asarray(a, np.float32) if case["precision"] == "mixed" else np.asarray(a)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "curve":
        out = pkg.run_curve(state["model"], *state["grid"], opts=state["opts"], ed=case["ed"])
        return {k: (v if case["ed"] else _as_held(case, v)) for k, v in out.items()}
    if kind == "train":
        net = E.Mlp(case["n_in"], case["width"], case["depth"], case["n_out"])
        net.set_params(state["p0"])
        hist = net.train(*state["data"], case["epochs"], case["batch"], case["lr"])
        out = {"params": net.get_params(), "loss": hist}
        net.close()
        return out
    eng, k = state["engine"], (case["mx"], case["my"])
    if kind == "apply":
        y = eng.block_apply(*k, state["x"])
        return y.astype(np.complex64) if case["precision"] == "mixed" else y
    eng.sector_prepare(case["nup"], case["ndn"])
    if kind == "spectrum":
        eng.blocks_ftlm_batched([k])
        ev, w, pref = eng.block_spectrum(*k, exact=False)
        return {"levels": _as_held(case, ev), "weights": _as_held(case, w), "prefactor": pref}
    eng.thermo_configure(*state["grid"])
    eng.blocks_ftlm_batched([k])
    eng.thermo_accumulate_block(*k)
    return {name: _as_held(case, a) for name, a in zip(("emin", "z", "n", "n2"), eng.thermo_read())}


# ------------------------------------------------------- what it cannot do without


def _ftlm_work(rows, hops, samples, steps, size):
    """Lanczos: 8 flops per hop and vector, ~30 per row of the recurrence; each step reads two vectors
    and writes one, unless they all stay on the chip."""
    steps = min(steps, max(rows, 1))
    vec = rows * samples * size
    return {"flops": rows * samples * steps * (8.0 * hops + 30.0),
            "bytes": 3.0 * vec * steps if 3 * vec > L2_BYTES else vec}


def work(case):
    kind = case["kind"]
    if kind == "train":
        sizes = [case["n_in"]] + [case["width"]] * case["depth"] + [case["n_out"]]
        par = sum(a * b for a, b in zip(sizes, sizes[1:]))
        rows = case["rows"] // case["batch"] * case["batch"] * case["epochs"]
        row_bytes = 4.0 * (case["n_in"] + 2 * case["n_out"])
        return {"flops": 6.0 * par * rows, "bytes": case["rows"] * row_bytes + 8.0 * par}
    size = 8 if case["precision"] == "mixed" else 16
    if kind == "apply":
        vec = _rows(case) * case["nvec"]
        return {"flops": vec * (8.0 * _hops(case) + 4), "bytes": 2.0 * 16 * vec}
    if kind in ("block", "spectrum"):
        return _ftlm_work(_rows(case), _hops(case), case["samples"], case["steps"], size)
    n = case["lx"] * case["ly"]
    w = {"flops": 0.0, "bytes": 0.0}
    for nup in range(n + 1):
        for ndn in range(n + 1):
            c = {**case, "nup": nup, "ndn": ndn}
            d = _rows(c)
            if case["ed"] or d <= case["threshold"]:
                w["flops"] += n * (16.0 / 3.0 * d ** 3 + 8 * d * _hops(c))
                w["bytes"] += n * 8 * d
            else:
                f = _ftlm_work(d, _hops(c), case["samples"], case["steps"], size)
                w["flops"] += n * f["flops"]
                w["bytes"] += n * f["bytes"]
    return w


# --------------------------------------------------------------- the same in 64 bits


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Spin:
    """Words of k particles on the lattice, their ranks, translations (rank and fermion sign) and hops."""

    def __init__(self, lx, ly, k):
        self.n = n = lx * ly
        dev = _dev()
        words = torch.arange(1 << n, dtype=torch.int64, device=dev)
        pop = sum((words >> s) & 1 for s in range(n))
        self.words = words[pop == k]
        self.rank = torch.full((1 << n,), -1, dtype=torch.int64, device=dev)
        self.rank[self.words] = torch.arange(len(self.words), device=dev)
        bits = [(self.words >> s) & 1 for s in range(n)]
        self.tr, self.tpar = [], []
        for s in range(n):
            to = [((q // lx + s // lx) % ly) * lx + (q % lx + s % lx) % lx for q in range(n)]
            self.tr.append(self.rank[sum(bits[q] << to[q] for q in range(n))])
            par = torch.zeros_like(self.words)
            for a in range(n):  # creation operators that change order
                for b in range(a + 1, n):
                    if to[a] > to[b]:
                        par ^= bits[a] & bits[b]
            self.tpar.append(par)

    def hop(self, a, b):
        """Ranks that can hop a -> b, where they land, and the parity of the particles passed."""
        w = self.words
        src = torch.nonzero(((w >> a) & 1 == 1) & ((w >> b) & 1 == 0)).flatten()
        w = w[src]
        par = torch.zeros_like(w)
        for s in range(min(a, b) + 1, max(a, b)):
            par ^= (w >> s) & 1
        return src, self.rank[w ^ (1 << a) ^ (1 << b)], par


class _Sector:
    """Translation orbits of a sector and every hop between their representatives (the smallest state of each)."""

    def __init__(self, m, nup, ndn):
        lx, ly, n = m.lx, m.ly, m.lx * m.ly
        self.m, self.n = m, n
        up, dn = _Spin(lx, ly, nup), _Spin(lx, ly, ndn)
        nd = len(dn.words)
        dev = up.words.device
        st = torch.arange(len(up.words) * nd, dtype=torch.int64, device=dev)
        best, shift, par = st.clone(), torch.zeros_like(st, dtype=torch.int8), torch.zeros_like(st, dtype=torch.int8)
        for s in range(1, n):  # T_s state = sign * image; the representative is the smallest image
            img = (up.tr[s][:, None] * nd + dn.tr[s][None, :]).flatten()
            p = (up.tpar[s][:, None] ^ dn.tpar[s][None, :]).flatten().to(torch.int8)
            less = img < best
            best[less], par[less], shift[less] = img[less], p[less], s
        self.reps = torch.nonzero(best == st).flatten()
        index = torch.full_like(st, -1)
        index[self.reps] = torch.arange(len(self.reps), device=dev)
        iu, jd = self.reps // nd, self.reps % nd
        stab = [(up.tr[s][iu] * nd + dn.tr[s][jd] == self.reps) for s in range(n)]
        self.stab = stab
        self.stab_sign = [1.0 - 2.0 * (up.tpar[s][iu] ^ dn.tpar[s][jd]).double() for s in range(n)]
        deg = sum(q.double() for q in stab)
        wu, wd = up.words[iu], dn.words[jd]
        occ = [((wu >> s) & 1) + ((wd >> s) & 1) for s in range(n)]
        nb = [[((q // lx + dy) % ly) * lx + (q % lx + dx) % lx for q in range(n)]
              for dx, dy in ((1, 0), (-1, 0), (0, 1), (0, -1), (1, 1), (-1, 1), (1, -1), (-1, -1))]
        bonds = [(q, nb[d][q]) for q in range(n) for d in (0, 2)]
        self.diag = m.u * sum(((wu >> s) & (wd >> s) & 1).double() for s in range(n)) + \
            m.v * sum((occ[a] * occ[b]).double() for a, b in bonds)
        thx, thy = 2 * math.pi * m.phix / lx, 2 * math.pi * m.phiy / ly
        ang = (thx, -thx, thy, -thy, thx + thy, thy - thx, thx - thy, -thx - thy)
        amp = (m.tx, m.tx, m.ty, m.ty, m.tp, m.tp, m.tp, m.tp)
        # hops by spin word, then spread over the representatives that hold it
        src, tgt, val, sft = [], [], [], []
        for spin, word, is_up in ((up, iu, True), (dn, jd, False)):
            where = torch.full((len(spin.words),), -1, dtype=torch.int64, device=dev)
            for d in range(8):
                if amp[d] == 0.0:
                    continue
                a = -amp[d] * complex(math.cos(ang[d]), math.sin(ang[d]))
                for q in range(n):
                    if nb[d][q] == q:
                        continue
                    r, to, p = spin.hop(q, nb[d][q])
                    if not len(r):
                        continue
                    where.fill_(-1)
                    where[r] = torch.arange(len(r), device=dev)
                    at = where[word]
                    i = torch.nonzero(at >= 0).flatten()
                    at = at[i]
                    moved = to[at] * nd + jd[i] if is_up else iu[i] * nd + to[at]
                    s0 = best[moved]
                    j = index[s0]
                    sign = 1.0 - 2.0 * (p[at] ^ par[moved].long()).double()
                    src.append(i)
                    tgt.append(j)
                    val.append(a * sign * torch.sqrt(deg[j] / deg[i]))
                    sft.append(shift[moved])
        cat = lambda v, t: torch.cat(v) if v else torch.zeros(0, dtype=t, device=dev)  # noqa: E731
        self.src, self.tgt = cat(src, torch.int64), cat(tgt, torch.int64)
        self.val, self.shift = cat(val, torch.complex128), cat(sft, torch.int8).long()

    def block(self, mx, my):
        """CSR of block (mx, my): rows are the representatives whose orbit sum does not vanish."""
        lx, ly = self.m.lx, self.m.ly
        ph = [complex(math.cos(t), math.sin(t)) for t in
              (2 * math.pi * (mx * (s % lx) / lx + my * (s // lx) / ly) for s in range(self.n))]
        amp = sum(self.stab[s].double() * self.stab_sign[s] * ph[s] for s in range(self.n))
        active = amp.abs() > 1e-9
        new = torch.cumsum(active.long(), 0) - 1
        dim = int(active.sum())
        keep = active[self.src] & active[self.tgt]
        # state = sign * T_{-shift} rep, so the hop carries e^{-i k.shift}
        back = torch.tensor([p.conjugate() for p in ph], dtype=torch.complex128, device=self.val.device)
        row, col = new[self.src[keep]], new[self.tgt[keep]]
        val = self.val[keep] * back[self.shift[keep]]
        own = torch.arange(dim, device=row.device)
        row, col = torch.cat([row, own]), torch.cat([col, own])
        val = torch.cat([val, self.diag[active].to(torch.complex128)])
        order = torch.argsort(row * max(dim, 1) + col)
        crow = torch.zeros(dim + 1, dtype=torch.int64, device=row.device)
        crow[1:] = torch.cumsum(torch.bincount(row, minlength=dim), 0) if dim else crow[1:]
        return dim, (row, col, val), torch.sparse_csr_tensor(crow, col[order], val[order], (dim, dim))


def _mix(v):
    M = (1 << 64) - 1
    v = (v + 0x9E3779B97F4A7C15) & M
    v = ((v ^ (v >> 30)) * 0xBF58476D1CE4E5B9) & M
    v = ((v ^ (v >> 27)) * 0x94D049BB133111EB) & M
    return v ^ (v >> 31)


def _block_seed(seed, nup, ndn, mx, my):
    s = _mix(seed)
    for v in (nup + 1, ndn + 17, mx + 257, my + 65537):
        s ^= _mix(v)
    return _mix(s)


def _philox(seed, dim, samples):
    """exp(2 pi i u)/sqrt(dim), u from Philox4x32-10 with counter (row, sample), key = the block seed."""
    dev, m32 = _dev(), 0xFFFFFFFF
    row = torch.arange(dim, dtype=torch.int64, device=dev)[:, None]
    c = [(row & m32).expand(dim, samples), (row >> 32).expand(dim, samples),
         torch.arange(samples, dtype=torch.int64, device=dev)[None, :].expand(dim, samples),
         torch.full((1, 1), 0x46544C4D, dtype=torch.int64, device=dev).expand(dim, samples)]
    k0, k1 = seed & m32, seed >> 32

    def mul(a, b):  # 32 x 32 -> (hi, lo) from 16-bit halves
        lo = a * (b & 0xFFFF)
        hi = a * (b >> 16) + (lo >> 16)
        return hi >> 16, ((hi & 0xFFFF) << 16) | (lo & 0xFFFF)

    for _ in range(10):
        h0, l0 = mul(c[0], 0xD2511F53)
        h1, l1 = mul(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
    u = (((c[0] << 21) ^ (c[1] >> 11)) & ((1 << 53) - 1)).double() / float(1 << 53)
    return torch.polar(torch.full_like(u, 1.0 / math.sqrt(dim)), 2 * math.pi * u)


def _mt64(seed, count):
    """`count` outputs of the 64-bit Mersenne twister (mt19937-64)."""
    M, nn, mm = (1 << 64) - 1, 312, 156
    s = [seed]
    for i in range(1, nn):
        s.append((6364136223846793005 * (s[-1] ^ (s[-1] >> 62)) + i) & M)
    s = np.array(s, np.uint64)
    up, low, a, one = np.uint64(M ^ 0x7FFFFFFF), np.uint64(0x7FFFFFFF), np.uint64(0xB5026F5AA96619E9), np.uint64(1)

    def twist(x, nxt, far):
        y = (x & up) | (nxt & low)
        return far ^ (y >> one) ^ np.where(y & one, a, np.uint64(0))

    out = []
    for _ in range(-(-count // nn)):
        s[:mm] = twist(s[:mm], s[1:mm + 1], s[mm:])
        s[mm:nn - 1] = twist(s[mm:nn - 1], s[mm + 1:], s[:nn - 1 - mm])
        s[nn - 1:] = twist(s[nn - 1:], s[:1], s[mm - 1:mm])
        out.append(s.copy())
    y = np.concatenate(out)[:count]
    y ^= (y >> np.uint64(29)) & np.uint64(0x5555555555555555)
    y ^= (y << np.uint64(17)) & np.uint64(0x71D67FFFEDA60000)
    y ^= (y << np.uint64(37)) & np.uint64(0xFFF7EEE000000000)
    return y ^ (y >> np.uint64(43))


def _gaussian(seed, dim, samples):
    """Unit-norm complex normals by the polar method: of each accepted pair (x, y) the y variate is drawn first;
    an element is (second draw, first draw)."""
    cols = []
    for v in range(samples):
        u = _mt64(_mix(seed ^ v), int(dim * 2.8) + 200).astype(np.float64) / float(1 << 64)
        u = 2.0 * u - 1.0
        x, y = u[0::2][:len(u) // 2], u[1::2][:len(u) // 2]
        r2 = x * x + y * y
        ok = np.nonzero((r2 <= 1.0) & (r2 != 0.0))[0][:dim]
        f = np.sqrt(-2.0 * np.log(r2[ok]) / r2[ok])
        q = x[ok] * f + 1j * (y[ok] * f)
        cols.append(q / np.linalg.norm(q))
    return torch.from_numpy(np.stack(cols, 1)).to(_dev())


def _ritz(h, q, steps):
    """Ritz values and first-component weights of plain Lanczos from each column of q."""
    dim, r = q.shape
    k = min(steps, dim)
    alpha, beta, last = torch.zeros(k, r), torch.zeros(k, r), [k] * r
    prev, bet = torch.zeros_like(q), torch.zeros(r, dtype=torch.float64, device=q.device)
    live = torch.ones(r, dtype=torch.bool, device=q.device)
    alpha, beta = alpha.double().to(q.device), beta.double().to(q.device)
    for j in range(k):
        w = h @ q
        a = (q.conj() * w).real.sum(0)
        w = w - a * q - bet * prev
        bet = torch.sqrt((w.real ** 2 + w.imag ** 2).sum(0))
        alpha[j], beta[j] = a, bet
        stop = live & (bet < 1e-12)
        for i in torch.nonzero(stop).flatten().tolist():
            last[i] = j + 1
        live &= ~stop
        prev, q = q, w / torch.where(bet < 1e-12, torch.ones_like(bet), bet)
    alpha, beta = alpha.cpu().numpy(), beta.cpu().numpy()
    out = []
    for i in range(r):
        s = last[i]
        e, v = np.linalg.eigh(np.diag(alpha[:s, i]) + np.diag(beta[:s - 1, i], 1) + np.diag(beta[:s - 1, i], -1))
        out.append((e, v[0] ** 2 / r))
    return np.concatenate([e for e, _ in out]), np.concatenate([w for _, w in out])


def _ftlm(case, seed, h, dim, nup, ndn, mx, my):
    bs = _block_seed(12345 + seed, nup, ndn, mx, my)
    q = (_philox if case["start"] == "philox" else _gaussian)(bs, dim, case["samples"])
    return _ritz(h, q, case["steps"])


def _add(acc, ev, w, particles, betas, mu):
    """Shifted Boltzmann sums of one spectrum."""
    for ib, b in enumerate(betas):
        low = ev.min() - mu * particles
        new = np.minimum(acc[0][ib], low)
        scale = np.where(np.isfinite(acc[0][ib]), np.exp(-b * np.where(np.isfinite(acc[0][ib]), acc[0][ib] - new, 0)), 0)
        z = (w[:, None] * np.exp(-b * (ev[:, None] - mu[None, :] * particles - new[None, :]))).sum(0)
        for p in range(3):
            acc[p + 1][ib] = acc[p + 1][ib] * scale + particles ** p * z
        acc[0][ib] = new


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return None  # the order of the mini-batches is the engine's own
    m = _model(case, seed)
    if kind == "curve":
        return _exact_curve(case, seed, m)
    if _rows(case) * (_hops(case) + 12) * case.get("samples", 1) * case.get("steps", 1) > 7e11:
        return None  # too long
    dim, _, h = _Sector(m, case["nup"], case["ndn"]).block(case["mx"], case["my"])
    if kind == "apply":
        y = h @ torch.from_numpy(_vectors(case, seed)).to(_dev())
        return y.cpu().numpy()
    ev, w = _ftlm(case, seed, h, dim, case["nup"], case["ndn"], case["mx"], case["my"])
    if kind == "spectrum":
        return {"levels": ev, "weights": w, "prefactor": float(dim)}
    betas, mu = _grid(case)
    acc = [np.full((len(betas), len(mu)), np.inf)] + [np.zeros((len(betas), len(mu))) for _ in range(3)]
    _add(acc, ev, dim * w, case["nup"] + case["ndn"], betas, mu)
    return dict(zip(("emin", "z", "n", "n2"), acc))


def _exact_curve(case, seed, m):
    betas, mu = _grid(case)
    n = m.sites
    acc = [np.full((len(betas), len(mu)), np.inf)] + [np.zeros((len(betas), len(mu))) for _ in range(3)]
    for nup in range(n + 1):
        for ndn in range(n + 1):
            sector = _Sector(m, nup, ndn)
            for k in range(n):
                mx, my = k % m.lx, k // m.lx
                dim, (row, col, val), h = sector.block(mx, my)
                if dim == 0:
                    continue
                if case["ed"] or dim <= case["threshold"]:
                    a = torch.zeros(dim * dim, dtype=torch.complex128, device=val.device)
                    a = a.index_add_(0, row * dim + col, val).view(dim, dim).cpu().numpy()
                    ev = np.linalg.eigvalsh(0.5 * (a + a.conj().T))
                    w = np.ones(dim)
                else:
                    ev, w = _ftlm(case, seed, h, dim, nup, ndn, mx, my)
                    w = dim * w
                _add(acc, ev, w, nup + ndn, betas, mu)
    emin, z, n1, n2 = acc
    b = np.asarray(betas).reshape(-1, 1)
    mean = n1 / z
    chi = np.maximum(0.0, (n2 / z - mean * mean) / n)
    return {"n": mean / n, "charge_correlation": chi, "compressibility": b * chi, "partition_like": z,
            "log_partition": np.log(z) - b * emin}
