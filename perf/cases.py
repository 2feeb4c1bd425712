"""Performance cases: the work that programs built on sfci_gb300 have it do.

Nearly all of a run's time is the SpMSpV product H v of a truncated vector, at
every length between the first Krylov vectors (one to a few thousand
determinants) and the truncation length Nd, so most cases are products: both
key widths, odd lengths, the shift and the capped output of MINRES, and sizes
from where latency counts to tens of GB of terms.  Beside them stand one whole
truncated Lanczos solve, the vector side of one Krylov step, calc_energy, the
linear solver's product and a training step and inference of the learned
screen.

Hamiltonians are the synthetic integrals of sfci_gb300.fcidump (20, 56 and 68
spin orbitals).  Vectors are shaped like the truncated Krylov vectors those
Hamiltonians give: determinants chosen by the excitation costs of their spin
strings plus noise, the Hartree-Fock determinant dominant, and magnitudes that
fall with the rank as a Krylov vector's do (0.98 for the first, 1e-2 for the
100th, 3e-5 for the 10,000th, 1.4e-6 for the 100,000th).
"""
import math
import os
import tempfile
from itertools import combinations

import numpy as np
import torch

import sfci_gb300 as sg
from sfci_gb300 import fcidump

# spatial orbitals, electrons and integral seed by spin orbitals: the small
# ground-state run, the benchmark's system, and a two-word system from inside
# the bond-stretch curve's range of 40 to 80 spin orbitals
SYSTEMS = {20: (10, 10, 0), 56: (28, 14, 1), 68: (34, 16, 4)}
CUT = 1e-5  # the default post-merge cut
# magnitude by rank of a truncated Krylov vector of the 56-spin-orbital system
RANKS = np.array([1.0, 10.0, 100.0, 1e3, 5e3, 1e4, 5e4, 1e5, 5e5, 1e6, 4e6])
MAGNITUDES = np.array([0.976, 3.0e-2, 1.15e-2, 3.2e-4, 1.05e-4, 3.0e-5, 2.6e-6, 1.4e-6, 1.9e-7, 7e-8, 1.5e-8])


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # the first Krylov vectors of any run, and every product of a small one
        product("product_20orb_64", 20, 64, keep=1500),
        # the truncation length of the 20-spin-orbital ground-state run
        product("product_20orb_20000", 20, 20000),
        # the growing vectors of the first steps on the benchmark's system
        product("product_56orb_3001", 56, 3001, keep=100000),
        # MINRES: shifted, scaled, the input cut to its top Nd and the output capped
        product("product_56orb_20000_shifted", 56, 20000, extra=7500, lam=-2.75, coeff=-0.5, cap=150000, keep=150000),
        # truncated steps of the benchmark's system: tens of GB of terms
        product("product_56orb_120000", 56, 120000),
        # two-word keys
        product("product_68orb_9001", 68, 9001, keep=50000),
        # a whole solve: one restart of the truncated Lanczos driver
        {"name": "lanczos_56orb_5000", "kind": "lanczos", "orb": 56, "nd": 5000, "nl": 6},
        # what a Krylov step does beside its product, on long vectors
        {"name": "krylov_vectors_1000003", "kind": "vectors", "orb": 56, "n": 1000003, "nd": 400000},
        # the energy of a truncated vector on its own support
        {"name": "energy_56orb_20011", "kind": "energy", "orb": 56, "n": 20011},
        # the linear (shift-invert) solver's product: dots with the basis, two vectors removed
        {"name": "linear_56orb_2500", "kind": "linear", "orb": 56, "n": 2500, "nb": 3},
        # the learned screen: gradients of one batch
        {"name": "screen_train_56orb", "kind": "train", "orb": 56, "n": 400, "tiles": 256},
        # and its inference on the term groups of a vector
        {"name": "screen_predict_56orb_1500", "kind": "predict", "orb": 56, "n": 1500},
    ]


def product(name, orb, nd, extra=0, lam=0.0, coeff=1.0, cap=2000000, keep=0):
    """One product of the top nd of a vector of nd + extra determinants, into a vector
    of capacity cap, truncated to its top keep (nd by default) as every Krylov step does."""
    case = {"kind": "product", "orb": orb, "nd": nd, "extra": extra, "lam": lam, "coeff": coeff, "cap": cap,
            "keep": keep or min(nd, cap)}
    return dict(case, name=name) if name else case


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product"] * 6 + ["lanczos", "vectors", "energy", "linear", "train", "predict"])
    if kind == "product":
        orb = rng.choice([20, 56, 56, 56, 68])
        nd = log_int(rng, 2, {20: 20000, 56: 120000, 68: 9001}[orb])
        if rng.random() < 0.3:
            return product(None, orb, nd, extra=rng.randrange(1, nd + 1), lam=round(rng.uniform(-4.0, 4.0), 3),
                           coeff=rng.choice([-1.0, -0.5, 0.25, 2.0]), cap=log_int(rng, 100, 2000000))
        return product(None, orb, nd)
    if kind == "lanczos":
        return {"kind": kind, "orb": rng.choice([20, 56]), "nd": log_int(rng, 500, 10000), "nl": rng.randrange(3, 9)}
    if kind == "vectors":
        n = log_int(rng, 1000, 1500000)
        return {"kind": kind, "orb": 56, "n": n, "nd": max(2, n // rng.randrange(1, 6))}
    if kind == "energy":
        return {"kind": kind, "orb": rng.choice([56, 56, 68]), "n": log_int(rng, 100, 30000)}
    if kind == "linear":
        return {"kind": kind, "orb": 56, "n": log_int(rng, 100, 5000), "nb": rng.randrange(1, 6)}
    if kind == "train":
        return {"kind": kind, "orb": 56, "n": rng.randrange(100, 500), "tiles": log_int(rng, 8, 512)}
    return {"kind": "predict", "orb": 56, "n": log_int(rng, 20, 2500)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def in_file(orb):
    """The system's _IN file, written once per machine."""
    M, ne, seed = SYSTEMS[orb]
    path = os.path.join(tempfile.gettempdir(), "sfci_perf_m%d_ne%d_s%d_IN" % (M, ne, seed))
    if not os.path.exists(path):
        tmp = "%s.%d" % (path, os.getpid())
        fcidump.rhf_to_in_file(tmp, M, ne, seed)
        os.remove(tmp + ".fcidump")
        os.replace(tmp, path)
    return path


def choose(items, e):
    return np.array(list(combinations(items, e)), np.int64).reshape(math.comb(len(items), e), e)


def spin_strings(M, n, rng):
    """Spin strings of n electrons up to a few excitations from the lowest, and their costs, ascending."""
    parts = []
    for e in range(min(4 if M <= 28 else 3, n, M - n) + 1):
        holes, into = choose(range(n), e), choose(range(n, M), e)
        flip = np.left_shift(1, holes).sum(1)[:, None] | np.left_shift(1, into).sum(1)[None, :]
        cost = 2.0 * e + 0.025 * (into.sum(1)[None, :] - holes.sum(1)[:, None])
        parts.append((((1 << n) - 1) ^ flip.ravel(), cost.ravel()))
    s, c = (np.concatenate(x) for x in zip(*parts))
    c[1:] += 0.5 * rng.standard_normal(len(c) - 1)
    order = np.argsort(c, kind="stable")
    return s[order], c[order]


def interleave(alpha, beta, M):
    """Determinant keys of spin strings: spatial orbital p is bits 2p (alpha) and 2p + 1 (beta)."""
    words = 1 if 2 * M <= 64 else 2
    key = np.zeros((len(alpha), words), np.uint64)
    for p in range(M):
        w, b = divmod(2 * p, 64)
        pair = ((alpha >> p) & 1) | (((beta >> p) & 1) << 1)
        key[:, w] |= pair.astype(np.uint64) << np.uint64(b)
    return key


def vector_parts(orb, n, seed):
    """Alpha strings, beta strings and amplitudes of a vector of n determinants, the largest first."""
    M, ne, _ = SYSTEMS[orb]
    rng = np.random.default_rng([seed, orb, n])
    (sa, ca), (sb, cb) = spin_strings(M, ne // 2, rng), spin_strings(M, ne // 2, rng)
    want = min(32 * n, len(sa) * len(sb))
    lo, hi = ca[0] + cb[0], ca[-1] + cb[-1]
    for _ in range(40):  # the cost under which `want` determinants lie
        mid = 0.5 * (lo + hi)
        if np.searchsorted(cb, mid - ca, side="right").sum() < want:
            lo = mid
        else:
            hi = mid
    per = np.searchsorted(cb, hi - ca, side="right")
    ia = np.repeat(np.arange(len(ca)), per)
    ib = np.arange(per.sum()) - np.repeat(np.cumsum(per) - per, per)
    score = ca[ia] + cb[ib] - 5.0 * rng.standard_normal(len(ia))
    score[(sa[ia] == sa.min()) & (sb[ib] == sb.min())] = -np.inf  # the Hartree-Fock determinant first
    n = min(n, len(score))
    best = np.argpartition(score, n - 1)[:n]
    best = best[np.argsort(score[best], kind="stable")]
    mag = np.exp(np.interp(np.log(np.arange(1, n + 1)), np.log(RANKS), np.log(MAGNITUDES)))
    mag *= rng.uniform(0.8, 1.2, n)
    amp = mag * np.where(rng.random(n) < 0.5, -1.0, 1.0)
    return sa[ia[best]], sb[ib[best]], amp / np.linalg.norm(amp)


def vector(orb, n, seed):
    """Keys and amplitudes of a vector of n determinants, keys ascending."""
    M = SYSTEMS[orb][0]
    alpha, beta, amp = vector_parts(orb, n, seed)
    key = interleave(alpha, beta, M)
    order = np.lexsort(tuple(key[:, w] for w in range(key.shape[1])))
    key, amp = key[order], amp[order]
    return (key[:, 0].copy() if key.shape[1] == 1 else key), amp


def context(orb, nd):
    M, ne, _ = SYSTEMS[orb]
    return sg.Context(in_file(orb), 2 * M, ne, Nd=nd, hpsi_cap=2000000)


def seeds(seed, n):
    return [int(s) for s in np.random.default_rng([seed, 77]).integers(1, 2 ** 31, n)]


def prepare(case, seed):
    orb, kind = case["orb"], case["kind"]
    ctx = context(orb, max(2, case.get("nd") or case["n"]))
    st = {"case": case, "ctx": ctx}
    if kind == "product":
        st["v"] = ctx.vec_from(*vector(orb, case["nd"] + case["extra"], seed))
        st["out"], st["kept"] = ctx.vec(case["cap"]), ctx.vec(case["keep"])
    elif kind == "lanczos":
        st["start"] = ctx.vec_from(*vector(orb, case["nd"] // 4, seed))
        st["v"] = ctx.vec(case["nd"])
    elif kind == "vectors":
        s = seeds(seed, 2)
        st["u"] = ctx.vec_from(*vector(orb, case["n"], s[0]))
        st["v"] = ctx.vec_from(*vector(orb, case["nd"], s[1]))
        st["t"], st["next"] = ctx.vec(case["n"] + case["nd"]), ctx.vec(case["nd"])
    elif kind == "energy":
        st["v"] = ctx.vec_from(*vector(orb, case["n"], seed))
    elif kind == "linear":
        s = seeds(seed, case["nb"])
        st["basis"] = [ctx.vec_from(*vector(orb, case["n"], x)) for x in s]
        st["out"], st["kept"] = ctx.vec(2000000), ctx.vec(case["n"])
    else:
        v = ctx.vec_from(*vector(orb, case["n"], seed))
        st["v"], st["screen"] = v, sg.Screen(ctx, seed=1 + seed % 1000)
        if kind == "train":
            out = ctx.vec(2000000)
            ctx.SpMVMtply_bucket(v, out, 0.0, 1.0)
            st["screen"].log(v, out, 1e-8)
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "product":
        diag = ctx.SpMVMtply_bucket(st["v"], st["out"], case["lam"], case["coeff"])
        st["kept"].shrinkFrom(st["out"])
        keys, amps = st["kept"].download()
        return {"keys": keys, "amps": amps, "diag": diag}
    if kind == "lanczos":
        st["v"].naiveCopy(st["start"])
        energies, energy = ctx.sparse_krylov_solve_eigenval(st["v"], case["nl"], 1)
        keys, amps = st["v"].download()
        return {"energies": energies, "energy": energy, "keys": keys, "amps": amps}
    if kind == "vectors":
        u, v, t, nxt = st["u"], st["v"], st["t"], st["next"]
        t.naiveCopy(u)
        t.addTwo(v, -0.37)
        nxt.shrinkFrom(t)
        norm = nxt.norm()
        nxt.scalarMtply(1.0 / norm)
        dot = v.dot(u)
        keys, amps = nxt.download()
        return {"norm": norm, "dot": dot, "keys": keys, "amps": amps}
    if kind == "energy":
        return {"energy": ctx.calc_energy(st["v"])}
    if kind == "linear":
        h = ctx.spmspvm_bucket_linear(st["basis"][-1], st["out"], 1.5, st["basis"])
        st["kept"].shrinkFrom(st["out"])
        keys, amps = st["kept"].download()
        return {"h": h, "keys": keys, "amps": amps}
    if kind == "train":
        loss = st["screen"].train(1, batch_tiles=case["tiles"], lr=0.0, pos_weight=2.0, sequential=True)
        return {"loss": loss, "grads": st["screen"].grads()}
    return {"prob": st["screen"].predict(st["v"], 0.01, probs=True)["prob"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def connected(orb):
    """Determinants connected to one, itself included."""
    M, ne, _ = SYSTEMS[orb]
    n, v = ne // 2, M - ne // 2
    pairs = math.comb(n, 2) * math.comb(v, 2)
    return 1 + 2 * n * v + 2 * pairs + (n * v) ** 2


def groups(orb):
    """Screened term groups of one determinant."""
    M, ne, _ = SYSTEMS[orb]
    n, v = ne // 2, M - ne // 2
    return 2 * math.comb(n, 2) * (v - 1) + n * v * n


def work(case):
    orb, kind = case["orb"], case["kind"]
    M = SYSTEMS[orb][0]
    entry = 16 if 2 * M <= 64 else 24
    C = connected(orb)
    tables = 8 * 4 * (M * (M + 1) // 2) ** 2  # the two-body integrals
    if kind == "product":  # a multiplication and an addition for each term
        return {"bytes": tables + entry * (case["nd"] + case["extra"] + case["keep"]),
                "flops": 2 * C * case["nd"]}
    if kind == "lanczos":  # nl products and the closing energy
        return {"bytes": tables + entry * 2 * case["nd"], "flops": 2 * C * case["nd"] * (case["nl"] + 1)}
    if kind == "vectors":
        return {"bytes": entry * (case["n"] + 2 * case["nd"]), "flops": 2 * (case["n"] + 3 * case["nd"])}
    if kind == "energy":
        return {"bytes": tables + entry * case["n"], "flops": 2 * C * case["n"]}
    if kind == "linear":
        return {"bytes": tables + entry * case["n"] * (case["nb"] + 1), "flops": 2 * C * case["n"]}
    layers = 576 * 256 + 256 * 256 + 256
    if kind == "train":
        rows = 128 * case["tiles"]
        return {"bytes": 4 * layers * 2 + 16 * rows, "flops": 6 * layers * rows}
    rows = groups(orb) * case["n"]
    return {"bytes": tables + 4 * rows + 4 * layers, "flops": 2 * layers * rows}


# ---------------------------------------------------------------------------
# the same results in 64 bits, without the framework's code
# ---------------------------------------------------------------------------

def exact(case, seed):
    orb, kind = case["orb"], case["kind"]
    if kind == "vectors":
        return exact_vectors(case, seed)
    if kind not in ("product", "energy", "linear") or 2 * SYSTEMS[orb][0] > 62:
        return None
    if connected(orb) * (case.get("nd") or case["n"]) > 7e8:
        return None
    h = Hamiltonian(orb)
    if kind == "product":
        keys, amps = vector(orb, case["nd"] + case["extra"], seed)
        keys, amps = largest(keys, amps, case["nd"])
        k, a = h.times(keys, amps, case["lam"], case["coeff"])
        diag = float(np.dot(amps, lookup(k, a, keys)))
        sel = np.abs(a) > CUT
        k, a = largest(k[sel], a[sel], min(case["cap"], case["keep"]))
        return {"keys": k, "amps": a, "diag": diag}
    if kind == "energy":
        keys, amps = vector(orb, case["n"], seed)
        k, a = h.times(keys, amps, 0.0, 1.0)
        return {"energy": float(np.dot(amps, lookup(k, a, keys)))}
    basis = [vector(orb, case["n"], x) for x in seeds(seed, case["nb"])]
    k, a = h.times(*basis[-1], 1.5, 1.0)
    hij = np.array([np.dot(amps, lookup(k, a, keys)) for keys, amps in basis])
    parts = [(k, a)] + [(basis[j][0], -hij[j] * basis[j][1]) for j in range(len(basis))[-2:]]
    k, inv = np.unique(np.concatenate([p[0] for p in parts]), return_inverse=True)
    a = np.zeros(len(k))
    np.add.at(a, inv, np.concatenate([p[1] for p in parts]))
    sel = np.abs(a) > CUT
    k, a = largest(k[sel], a[sel], case["n"])
    return {"h": hij, "keys": k, "amps": a}


def exact_vectors(case, seed):
    s = seeds(seed, 2)
    (ku, au), (kv, av) = vector(case["orb"], case["n"], s[0]), vector(case["orb"], case["nd"], s[1])
    k, inv = np.unique(np.concatenate([ku, kv]), return_inverse=True)
    a = np.zeros(len(k))
    np.add.at(a, inv, np.concatenate([au, -0.37 * av]))
    k, a = largest(k, a, case["nd"])
    norm = math.sqrt(math.fsum(a * a))
    return {"norm": norm, "dot": math.fsum(av * lookup(ku, au, kv)), "keys": k, "amps": a * (1.0 / norm)}


def largest(keys, amps, n):
    """The n entries of largest magnitude, in key order; of equal ones the highest keys."""
    if len(amps) <= n:
        return keys, amps
    sel = np.sort(np.argsort(np.abs(amps), kind="stable")[-n:])
    return keys[sel], amps[sel]


def lookup(keys, amps, of):
    i = np.minimum(np.searchsorted(keys, of), len(keys) - 1)
    return np.where(keys[i] == of, amps[i], 0.0)


class Hamiltonian:
    """Matrix elements of a synthetic RHF system between determinants of one 64-bit word."""

    def __init__(self, orb):
        M, ne, seed = SYSTEMS[orb]
        self.M, self.n = M, ne // 2
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        h, (i, j, k, l), v, _ = fcidump.synthetic_rhf(M, seed)
        g = np.zeros((M,) * 4)
        for p in ((i, j, k, l), (j, i, k, l), (i, j, l, k), (j, i, l, k),
                  (k, l, i, j), (k, l, j, i), (l, k, i, j), (l, k, j, i)):
            g[p] = v
        self.h, self.g = torch.from_numpy(h).to(self.dev), torch.from_numpy(g).to(self.dev)

    def parity(self, key, p, q):
        """Parity of the electrons strictly between spin orbitals p and q."""
        lo, hi = torch.minimum(p, q), torch.maximum(p, q)
        one = torch.ones_like(lo)
        x = key & ((one << hi) - 1) & ~((one << (lo + 1)) - 1)
        for s in (32, 16, 8, 4, 2, 1):
            x = x ^ (x >> s)
        return x & 1

    def move(self, key, src, dst):
        one = torch.ones_like(src)
        return key ^ (one << src) ^ (one << dst), self.parity(key, src, dst)

    def terms(self, key, lam):
        """Targets and elements of <target| H - lam |key> for a batch of determinants."""
        M, n, h, g = self.M, self.n, self.h, self.g
        bits = (key[:, None] >> torch.arange(2 * M, device=self.dev)) & 1
        occ = [torch.nonzero(bits[:, s::2] == 1)[:, 1].view(-1, n) for s in (0, 1)]
        vir = [torch.nonzero(bits[:, s::2] == 0)[:, 1].view(-1, M - n) for s in (0, 1)]
        up = [torch.tensor(list(combinations(range(m), 2)), device=self.dev).view(-1, 2).t() for m in (n, M - n)]
        out_k, out_v = [], []
        d = h[occ[0], occ[0]].sum(1) + h[occ[1], occ[1]].sum(1)
        for s in (0, 1):
            for t in (0, 1):
                a, b = occ[s][:, :, None], occ[t][:, None, :]
                d = d + 0.5 * g[a, a, b, b].sum((1, 2))
                if s == t:
                    d = d - 0.5 * g[a, b, b, a].sum((1, 2))
        out_k.append(key[:, None])
        out_v.append((d - lam)[:, None])
        for s in (0, 1):
            i, a = occ[s][:, :, None], vir[s][:, None, :]
            v = h[a, i]
            for t in (0, 1):
                k = occ[t][:, None, None, :]
                v = v + g[a[..., None], i[..., None], k, k].sum(-1)
                if s == t:
                    v = v - g[a[..., None], k, k, i[..., None]].sum(-1)
            i, a = torch.broadcast_tensors(i, a)
            k, par = self.move(key[:, None, None], 2 * i + s, 2 * a + s)
            out_k.append(k.flatten(1))
            out_v.append(torch.where(par == 1, -v, v).flatten(1))
            i, j = (occ[s][:, up[0][x]][:, :, None] for x in (0, 1))
            a, b = (vir[s][:, up[1][x]][:, None, :] for x in (0, 1))
            v = g[a, i, b, j] - g[b, i, a, j]
            i, j, a, b = torch.broadcast_tensors(i, j, a, b)
            k, p1 = self.move(key[:, None, None], 2 * i + s, 2 * a + s)
            k, p2 = self.move(k, 2 * j + s, 2 * b + s)
            out_k.append(k.flatten(1))
            out_v.append(torch.where(p1 ^ p2 == 1, -v, v).flatten(1))
        i, a = occ[0][:, :, None, None, None], vir[0][:, None, :, None, None]
        j, b = occ[1][:, None, None, :, None], vir[1][:, None, None, None, :]
        v = g[a, i, b, j]
        i, a, j, b = torch.broadcast_tensors(i, a, j, b)
        k, p1 = self.move(key[:, None, None, None, None], 2 * i, 2 * a)
        k, p2 = self.move(k, 2 * j + 1, 2 * b + 1)
        out_k.append(k.flatten(1))
        out_v.append(torch.where(p1 ^ p2 == 1, -v, v).flatten(1))
        return torch.cat(out_k, 1), torch.cat(out_v, 1)

    def times(self, keys, amps, lam, coeff):
        """Merged coeff (H - lam) v: keys ascending, amplitudes."""
        key = torch.from_numpy(keys.astype(np.int64)).to(self.dev)
        amp = torch.from_numpy(amps).to(self.dev) * coeff
        got_k, got_v = [], []
        for at in range(0, len(amps), 256):
            k, v = self.terms(key[at:at + 256], lam)
            got_k.append(k.flatten())
            got_v.append((v * amp[at:at + 256, None]).flatten())
        k, inv = torch.unique(torch.cat(got_k), return_inverse=True)
        out = torch.zeros(len(k), dtype=torch.float64, device=self.dev)
        out.index_add_(0, inv, torch.cat(got_v))
        return k.cpu().numpy().astype(np.uint64), out.cpu().numpy()
