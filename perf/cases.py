"""Timed cases of the engine: the calls a host program makes, over the sizes it makes them at.

A case names a kind of call, a system (norb, na, nb: spatial orbitals, alpha and beta electrons), a
target number of determinants and the call's options. Systems have the integrals of the molecular
family of this repository's workloads (mol10 ... mol50: h_pp sorted in [-2, 2], h_pq ~ N(0, 0.05),
Cholesky vectors ~ N(0, 0.1) exp(-|p-q|/6)), one fixed set per norb, or of the Hubbard ring. The
determinant spaces are those of a selected CI run, found with the engine's own selection: from the
lowest determinant, then from that space with first-order coefficients. The seed
gives the order of the determinants, the coefficients and the vectors.

Kinds:
  run       shci_run_input, the whole variational stage of an input file (the 12-site ring)
  sigma     y = H x on the stored or the matrix-free Hamiltonian; call = host (numpy vectors, as a
            CPU driver's Davidson passes them), device (column-major FP64 vectors on the GPU) or
            packed (the engine's gather layout)
  grow      one step of the schedule: Hamiltonian of a space, selection, Hamiltonian of the grown
            space (the stored rows extended), one sigma on it
  select    heat-bath selection from every determinant of a space
  davidson  one eigensolve from the reference determinant
  pt        deterministic second-order correction
  ptstoch   a fixed number of iterations of the semistochastic correction
  rdm       spatial 1- and 2-RDM of a vector on a stored Hamiltonian
"""
import functools
import math
import os
import tempfile

import numpy as np
import torch

from dice_gb300 import engine


# ---- cases ------------------------------------------------------------------
def listed():
    return [
        # a small calculation from input file to energy: parser, tables, six selections, Davidson
        dict(name="run_hubbard12", kind="run", norb=12, na=6, nb=6, ndets=68000, eps1=1e-4, iters=6),
        # the smallest sigma calls: a CPU driver's own Davidson on a few thousand determinants
        dict(name="sigma_host_small", kind="sigma", norb=10, na=4, nb=4, ndets=4000, mode="fp64", k=1, call="host"),
        # the plain FP64 path's sigma at an ordinary size
        dict(name="sigma_fp64", kind="sigma", norb=24, na=12, nb=12, ndets=250000, mode="fp64", k=1, call="device"),
        # the mixed path's sigma at the largest space
        dict(name="sigma_mixed_large", kind="sigma", norb=24, na=12, nb=12, ndets=1200000, mode="mixed", k=1,
             call="packed"),
        # block Davidson of four roots, two-word determinants
        dict(name="sigma_block4", kind="sigma", norb=36, na=14, nb=14, ndets=200000, mode="mixed", k=4, call="packed"),
        # the matrix-free path, four roots
        dict(name="sigma_direct4", kind="sigma", norb=36, na=14, nb=14, ndets=100000, mode="direct", k=4,
             call="device"),
        # one step of the schedule in the mixed form
        dict(name="grow_mixed", kind="grow", norb=24, na=12, nb=12, ndets=400000, mode="mixed"),
        # selection from an odd-electron two-word space
        dict(name="select", kind="select", norb=36, na=14, nb=13, ndets=60000, grow=4.0),
        # one Davidson solve at an ordinary size
        dict(name="davidson", kind="davidson", norb=24, na=12, nb=12, ndets=80000, mode="fp64", roots=1),
        # deterministic PT2 of an ordinary variational space
        dict(name="pt", kind="pt", norb=24, na=12, nb=12, ndets=80000, eps2=2e-5),
        # semistochastic PT2: many small iterations
        dict(name="ptstoch", kind="ptstoch", norb=24, na=12, nb=12, ndets=80000, eps2=1e-6, sample=200, iters=10),
        # density matrices after a variational run
        dict(name="rdm", kind="rdm", norb=24, na=12, nb=12, ndets=150000, mode="mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sigma", "sigma", "sigma", "sigma", "grow", "select", "davidson", "pt", "ptstoch", "rdm", "run"])
    if kind == "run":
        n = rng.choice([8, 10, 12])
        return dict(kind="run", norb=n, na=n // 2, nb=n // 2, ndets=68000 if n == 12 else 10000,
                    eps1=round(math.exp(rng.uniform(math.log(1e-4), math.log(3e-3))), 6), iters=rng.randint(3, 6))
    n = rng.choice([10, 13, 16, 20, 24, 24, 27, 32, 33, 36, 40, 50])
    na = max(3, int(n * rng.uniform(0.32, 0.5)))
    nb = max(3, na - rng.choice([0, 0, 0, 1, 2]))
    # the determinants with up to two electrons moved twice bound what a small system can hold
    full = math.comb(n, na) * math.comb(n, nb)
    c = dict(kind=kind, norb=n, na=na, nb=nb)
    if kind == "sigma":
        mode = rng.choice(["fp64", "mixed", "mixed", "refine", "direct", "direct_mixed"])
        top = 100000 if mode.startswith("direct") else 700000
        c.update(ndets=_log(rng, 500, min(top, full // 4)), mode=mode, k=rng.choice([1, 1, 2, 3, 4]),
                 call=rng.choice(["host", "device", "packed"] if mode in ("fp64", "mixed") else ["host", "device"]))
    elif kind == "grow":
        c.update(ndets=_log(rng, 1000, min(300000, full // 4)), mode=rng.choice(["fp64", "mixed"]))
    elif kind == "select":
        c.update(ndets=_log(rng, 500, min(60000, full // 20)), grow=round(rng.uniform(1.5, 4.0), 2))
    elif kind == "davidson":
        c.update(ndets=_log(rng, 500, min(60000, full // 4)), mode=rng.choice(["fp64", "fp64", "direct"]),
                 roots=rng.choice([1, 1, 2]))
        if c["mode"] == "direct":
            c["ndets"] = max(500, c["ndets"] // 8)
    elif kind in ("pt", "ptstoch"):
        c.update(ndets=_log(rng, 500, min(60000, full // 20)),
                 eps2=round(math.exp(rng.uniform(math.log(2e-5), math.log(1e-3))), 7))
        if kind == "ptstoch":
            c.update(sample=rng.choice([100, 200, 500]), iters=rng.randint(4, 10))
    else:
        c.update(ndets=_log(rng, 500, min(100000, full // 4)), mode=rng.choice(["fp64", "mixed"]))
    return c


# ---- systems and spaces -------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _integrals(n):
    rng = np.random.default_rng(20260000 + n)
    h = np.triu(rng.normal(0.0, 0.05, size=(n, n)), 1)
    h = h + h.T
    h[np.diag_indices(n)] = np.sort(rng.uniform(-2.0, 2.0, size=n))
    p = np.arange(n)
    L = np.triu(rng.normal(0.0, 0.1, size=(3 * n, n, n)))
    L = (L + np.transpose(np.triu(L, 1), (0, 2, 1))) * np.exp(-np.abs(p[:, None] - p) / 6.0)
    L = L.reshape(3 * n, n * n)
    eri = (L.T @ L).reshape(n, n, n, n)
    for _ in range(2):  # symmetric in every bit: each class takes the value that the file holds
        eri = np.maximum(eri, eri.transpose(1, 0, 2, 3))
        eri = np.maximum(eri, eri.transpose(0, 1, 3, 2))
        eri = np.maximum(eri, eri.transpose(2, 3, 0, 1))
    return h, eri


def _ring(n, u):
    h = np.zeros((n, n))
    for i in range(n):
        h[i, (i + 1) % n] = h[(i + 1) % n, i] = -1.0
    eri = np.zeros((n, n, n, n))
    eri[np.arange(n), np.arange(n), np.arange(n), np.arange(n)] = u
    return h, eri


def _write_fcidump(path, h, eri, na, nb):
    n = len(h)
    P, Q = np.tril_indices(n)
    A, B = np.tril_indices(len(P))
    two = eri[P[A], Q[A], P[B], Q[B]]
    keep = np.nonzero(two)[0]
    A, B = A[keep], B[keep]
    rows = ["%.17g %d %d %d %d" % r for r in zip(two[keep].tolist(), (P[A] + 1).tolist(), (Q[A] + 1).tolist(),
                                                 (P[B] + 1).tolist(), (Q[B] + 1).tolist())]
    rows += ["%.17g %d %d 0 0" % (h[p, q], p + 1, q + 1) for p, q in zip(P, Q) if h[p, q] != 0.0]
    with open(path, "w") as f:
        f.write(" &FCI NORB=%d,NELEC=%d,MS2=%d,\n  ORBSYM=%s\n  ISYM=1,\n &END\n" % (n, na + nb, na - nb, "1," * n))
        f.write("\n".join(rows) + "\n0.0 0 0 0 0\n")


@functools.lru_cache(maxsize=None)
def _fcidump(n, na, nb):
    path = os.path.join(tempfile.mkdtemp(prefix="shci_cases_"), "FCIDUMP")
    _write_fcidump(path, *_integrals(n), na, nb)
    return path


def _spread(x):
    """Bit k of each string to bit 2k of a pair of words (uint64)."""
    lo, hi = x & np.uint64(0xffffffff), x >> np.uint64(32)
    out = []
    for v in (lo, hi):
        for s, m in ((16, 0x0000ffff0000ffff), (8, 0x00ff00ff00ff00ff), (4, 0x0f0f0f0f0f0f0f0f),
                     (2, 0x3333333333333333), (1, 0x5555555555555555)):
            v = (v | (v << np.uint64(s))) & np.uint64(m)
        out.append(v)
    return np.stack(out, -1)


def _compact(w):
    out = []
    for v in (w[..., 0], w[..., 1]):
        v = v & np.uint64(0x5555555555555555)
        for s, m in ((1, 0x3333333333333333), (2, 0x0f0f0f0f0f0f0f0f), (4, 0x00ff00ff00ff00ff),
                     (8, 0x0000ffff0000ffff), (16, 0x00000000ffffffff)):
            v = (v | (v >> np.uint64(s))) & np.uint64(m)
        out.append(v)
    return out[0] | (out[1] << np.uint64(32))


def _strings(dets):
    """Alpha and beta strings of determinants (spin orbital 2k + s is spatial orbital k)."""
    return _compact(dets), _compact(dets >> np.uint64(1))


def _noise(dets, seed, width):
    """A factor between exp(-width) and exp(width) per determinant, the same for an alpha <-> beta flipped pair."""
    a, b = _strings(dets)
    x = (np.minimum(a, b) * np.uint64(0x9e3779b97f4a7c15)) ^ (np.maximum(a, b) + np.uint64(seed * 2 + 1))
    for _ in range(3):
        x = (x ^ (x >> np.uint64(31))) * np.uint64(0xbf58476d1ce4e5b9)
    x ^= x >> np.uint64(29)
    return np.exp(width * 2.0 * ((x >> np.uint64(11)).astype(np.float64) / 2.0 ** 53 - 0.5))


def _grown(e, dets, cmax, target):
    """The space selection from `dets` gives with the threshold that brings it to about `target`."""
    def size(eps):
        e.set_dets(dets)
        e.select(cmax, eps)
        return e.ndets()

    hi = 3e-2
    while (n := size(hi)) < target and hi > 1e-7:
        lo, hi = hi, hi / 2
    if n >= target and hi < 3e-2:
        lo, hi = hi, 2 * hi
        for _ in range(5):
            mid = math.sqrt(lo * hi)
            lo, hi = (mid, hi) if size(mid) >= target else (lo, mid)
        eps = lo
    else:
        eps = hi
    size(eps)
    return e.dets(), eps


def _first_order(e, dets, c):
    """Coefficients of `dets` to first order in the vector c of its first determinants."""
    e.set_dets(dets)
    e.ham_build("fp64")
    x = np.zeros(len(dets))
    x[:len(c)] = c
    y, diag = e.sigma(x, "fp64"), e.diag()
    e0 = float(x @ y) / float(x @ x)
    out = y / np.minimum(e0 - diag, -0.05)
    out[:len(c)] = c
    # 24 bits are kept, so that the last bits of a sum do not matter to a selection from them
    out = out.astype(np.float32).astype(np.float64)
    return out / np.abs(out).max()


@functools.lru_cache(maxsize=16)
def _space(norb, na, nb, target, coefficients):
    """A selected space of about `target` determinants, the lowest one first, and, where asked for, its
    coefficients (largest one 1)."""
    e = engine.Engine(0)
    e.read_fcidump(_fcidump(norb, na, nb))
    a, b = np.uint64((1 << na) - 1), np.uint64((1 << nb) - 1)
    ref = (_spread(a) | (_spread(b) << np.uint64(1))).reshape(1, 2)
    s1, _ = _grown(e, ref, np.ones(1), max(50, target // 5))
    c1 = _first_order(e, s1, np.ones(1)) * _noise(s1, norb, 0.5)
    c1[0] = 1.0
    dets, _ = _grown(e, s1, np.abs(c1), target)
    c = _first_order(e, dets, c1) if coefficients else None
    e.close()
    return dets, c


def _ordered(v, seed):
    """The same space met in another order: all but the first entry rolled by an amount that the seed gives."""
    n = max(1, len(v) - 1)
    return np.ascontiguousarray(np.concatenate([v[:1], np.roll(v[1:], (seed * 7919 + 13) % n, axis=0)]))


def _vectors(seed, k, n):
    """Unit vectors with entries over several decades, as a Davidson basis has them."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(k, n, generator=g, device="cuda", dtype=torch.float64)
    x *= torch.exp(1.5 * torch.randn(k, n, generator=g, device="cuda", dtype=torch.float64))
    return x / x.norm(dim=1, keepdim=True)


# ---- one case -----------------------------------------------------------------
def _ring_input(case, seed):
    n, u = case["norb"], 4.0 + 0.2 * ((seed * 2654435761) % 1000) / 1000.0
    where = tempfile.mkdtemp(prefix="shci_run_")
    _write_fcidump(os.path.join(where, "FCIDUMP"), *_ring(n, u), case["na"], case["nb"])
    occ = sorted([2 * s for s in range(0, n, 2)][:case["na"]] + [2 * s + 1 for s in range(1, n, 2)][:case["nb"]])
    with open(os.path.join(where, "input.dat"), "w") as f:
        f.write("nocc %d\n%s\nend\norbitals FCIDUMP\nnroots 1\nschedule\n0 1e-2\n%d %g\nend\n"
                "davidsonTol 1e-9\ndavidsonTolLoose 1e-7\ndE 1e-10\nmaxiter %d\nnoio\n"
                % (len(occ), " ".join(map(str, occ)), case["iters"] // 2, case["eps1"], case["iters"]))
    return os.path.join(where, "input.dat")


def prepare(case, seed):
    e = engine.Engine(0)
    s = dict(case=case, e=e)
    kind = case["kind"]
    if kind == "run":
        s["input"] = _ring_input(case, seed)
        return s
    size = case["norb"], case["na"], case["nb"], case["ndets"]
    e.read_fcidump(_fcidump(*size[:3]))
    if kind == "sigma":
        dets = _ordered(_space(*size, False)[0], seed)
        n, k, mode = len(dets), case["k"], case["mode"]
        x = _vectors(seed, k, n)
        e.set_dets(dets)
        e.ham_build("mixed" if mode == "refine" else mode)
        s.update(n=n, dets=dets, mode="fp64" if mode == "refine" else mode)
        if case["call"] == "host":
            s["x"] = x.cpu().numpy()
        elif case["call"] == "device":
            s["x"] = x
        else:
            kp = 4 if k == 3 else k
            p = torch.zeros(n, kp, device="cuda", dtype=torch.float32 if mode == "mixed" else torch.float64)
            p[:, :k] = x.T
            s.update(x=p, kp=kp)
        s["y"] = torch.zeros(k, n, device="cuda", dtype=torch.float64)
    elif kind == "grow":
        small, c = (_ordered(v, seed) for v in _space(*size[:3], max(200, case["ndets"] // 5), True))
        grown, eps = _grown(e, small, np.abs(c), case["ndets"])
        s.update(small=small, cmax=np.abs(c), eps=eps, n=len(grown), x=_vectors(seed, 1, len(grown)))
        s["y"] = torch.zeros(1, len(grown), device="cuda", dtype=torch.float64)
    elif kind == "select":
        dets, c = (_ordered(v, seed) for v in _space(*size, True))
        _, eps = _grown(e, dets, np.abs(c), int(case["grow"] * len(dets)))
        s.update(dets=dets, cmax=np.abs(c), eps=eps)
    elif kind == "davidson":
        dets = _ordered(_space(*size, False)[0], seed)
        x0 = np.zeros((case["roots"], len(dets)))
        x0[0, 0] = 1.0
        e.set_dets(dets)
        e.ham_build(case["mode"])
        s.update(dets=dets, x0=x0)
    else:
        dets, c = (_ordered(v, seed) for v in _space(*size, True))
        c *= _noise(dets, seed, 0.5)
        c /= np.linalg.norm(c)
        e.set_dets(dets)
        # a variational energy of such a space: some 0.15 per orbital below its lowest determinant
        s.update(dets=dets, c=c, e0=float(e.diag().min()) - 0.15 * case["norb"], seed=1 + seed % 1000)
        if kind == "rdm":
            e.ham_build(case["mode"])
    return s


def run(s):
    case, e = s["case"], s["e"]
    kind = case["kind"]
    if kind == "run":
        E = e.run_input(s["input"], mode="fp64")
        return {"E": E, "ndets": e.run_log()["ndets"], "dets": e.dets().view(np.int64), "ci": e.run_ci(1)}
    if kind == "sigma":
        k, n = case["k"], s["n"]
        if case["call"] == "host":
            return e.sigma(s["x"], s["mode"])
        if case["call"] == "device":
            e.sigma_device(s["x"].data_ptr(), s["y"].data_ptr(), k, n, s["mode"])
        else:
            e.sigma_packed_device(s["x"].data_ptr(), s["kp"], k, s["y"].data_ptr(), n, s["mode"])
        return s["y"]
    if kind == "grow":
        e.set_dets(s["small"])
        nnz0 = e.ham_build(case["mode"])
        e.select(s["cmax"], s["eps"])
        nnz1 = e.ham_build(case["mode"])
        e.sigma_device(s["x"].data_ptr(), s["y"].data_ptr(), 1, s["n"], case["mode"])
        return {"nnz": [nnz0, nnz1], "dets": e.dets().view(np.int64), "y": s["y"]}
    if kind == "select":
        e.set_dets(s["dets"])
        n = e.select(s["cmax"], s["eps"])
        return {"new": n, "dets": e.dets().view(np.int64)}
    if kind == "davidson":
        E, x, it = e.davidson(s["x0"], mode=case["mode"], tol=1e-7)
        return {"E": E, "x": x, "iterations": it}
    if kind == "pt":
        e2 = e.pt_deterministic(s["c"], s["e0"], case["eps2"])
        st = e.pt_stats()
        return {"e2": e2, "candidates": st["candidates"], "unique": st["unique"], "norm": st["psi1_norm"]}
    if kind == "ptstoch":
        e2, err, it = e.pt_semistochastic(s["c"], s["e0"], case["eps2"], sample_n=case["sample"],
                                          max_iter=case["iters"], target_error=1e-12, seed=s["seed"])
        return {"e2": e2, "error": err, "iterations": it}
    s2, s1 = e.rdm(s["c"])
    return {"two": s2, "one": s1}


# Measured off-diagonal entries per row of such spaces: 1171 (norb 24, 250,000 determinants), 1687 (24,
# 1.2 million), 1349 (36, 200,000), 280 (10, 4,000).
def _per_row(case):
    n, N = case["norb"], case["ndets"]
    if case["kind"] == "run":
        return 30.0
    return min(0.5 * N, 900.0 * (N / 1e5) ** 0.25 * min(1.25, 0.4 + 0.6 * n / 24))


def work(case):
    """Inputs read once and outputs written once; an entry of the stored matrix is a column and a value
    (2 + 4 bytes in the mixed form, whose columns ascend within a row, 4 + 8 in FP64), a matrix-free
    connection its two determinants' share (nothing beyond reading the space)."""
    N, kind = float(case["ndets"]), case["kind"]
    nnz = N * _per_row(case)
    ent = {"fp64": 12.0, "mixed": 6.0, "refine": 10.0}.get(case.get("mode"), 0.0)
    if kind == "run":
        return {"bytes": case["iters"] * (60.0 * 12.0 * nnz / 4 + 400.0 * N), "flops": case["iters"] * 30.0 * nnz}
    if kind == "sigma":
        k = case["k"]
        flops = 2.0 * nnz * k + (20.0 * nnz if case["mode"].startswith("direct") else 0.0)
        return {"bytes": nnz * ent + N * (8.0 + 16.0 * k) + (16.0 * N if ent == 0 else 0.0), "flops": flops}
    if kind == "grow":  # the matrix written once, read once by the sigma
        return {"bytes": nnz * (12.0 + ent) + 60.0 * N, "flops": 22.0 * nnz}
    if kind == "select":
        return {"bytes": N * (24.0 + 16.0 * case["grow"] * 2), "flops": 10.0 * N * case["grow"]}
    if kind == "davidson":
        its = 20.0 * case["roots"]
        return {"bytes": its * (nnz * ent + 200.0 * N), "flops": its * (2.0 * nnz + 80.0 * N)}
    if kind == "pt":  # a candidate's key and numerator, written and read once
        cand = N * 800.0 * min(1.0, 2e-5 / case["eps2"])
        return {"bytes": 2 * 32.0 * cand + 24.0 * N, "flops": 40.0 * cand}
    if kind == "ptstoch":
        cand = case["iters"] * case["sample"] * 3000.0
        return {"bytes": 2 * 32.0 * cand + 24.0 * N, "flops": 60.0 * cand}
    return {"bytes": nnz / 2 * 4.0 + 24.0 * N, "flops": 40.0 * nnz / 2}


# ---- the same in 64 bits --------------------------------------------------------
def _pop(x):
    x = x - ((x >> 1) & 0x5555555555555555)
    x = (x & 0x3333333333333333) + ((x >> 2) & 0x3333333333333333)
    x = (x + (x >> 4)) & 0x0f0f0f0f0f0f0f0f
    return (x * 0x0101010101010101) >> 56


def _low(x):
    """Index of the lowest set bit."""
    return _pop((x & -x) - 1)


class _Exact:
    """Slater-Condon elements between determinants given as alpha and beta strings (int64 tensors)."""

    def __init__(self, dets, n):
        a, b = _strings(dets)
        h, eri = _integrals(n)
        self.n, self.N = n, len(dets)
        self.s = [torch.from_numpy(v.astype(np.int64)).cuda() for v in (a, b)]
        self.h, self.eri = torch.from_numpy(h).cuda(), torch.from_numpy(eri).cuda()
        k = torch.arange(n, device="cuda")
        self.occ = [((v[:, None] >> k) & 1).double() for v in self.s]
        self.coul = self.eri[:, :, k, k].contiguous()              # (ai|jj)
        self.exch = self.eri[:, k, k, :].permute(0, 2, 1).contiguous()  # (aj|ji) at [a, i, j]
        J, K = self.coul[k, k], self.exch[k, k]
        oa, ob = self.occ
        t = oa + ob
        self.diag = (t @ torch.diagonal(self.h)) + 0.5 * ((t @ J * t).sum(1) - (oa @ K * oa).sum(1) - (ob @ K * ob).sum(1))

    @staticmethod
    def _below(a, b, p):
        """Occupied spin orbitals below spin orbital p."""
        one = torch.ones_like(p)
        return _pop(a & ((one << ((p + 1) // 2)) - 1)) + _pop(b & ((one << (p // 2)) - 1))

    def _sign(self, a, b, i, o):
        """Parity of moving an electron from spin orbital i to o."""
        return (self._below(a, b, torch.maximum(i, o)) - self._below(a, b, torch.minimum(i, o)) - (i < o).long()) & 1

    def elements(self, r, c, da, db):
        """H[r, c] for connected pairs whose alpha and beta strings differ by da and db bits."""
        out = torch.zeros(len(r), dtype=torch.float64, device="cuda")
        for sp in (0, 1):
            ds, do = (da, db) if sp == 0 else (db, da)
            m = torch.nonzero((ds == 2) & (do == 0))[:, 0]
            if len(m):
                R, C = r[m], c[m]
                x, y = self.s[sp][R], self.s[sp][C]
                o, i = _low(x & ~y), _low(y & ~x)
                v = self.h[o, i] + (self.occ[sp][C] * (self.coul[o, i] - self.exch[o, i])).sum(1) \
                    + (self.occ[1 - sp][C] * self.coul[o, i]).sum(1)
                sg = self._sign(self.s[0][C], self.s[1][C], 2 * i + sp, 2 * o + sp)
                out[m] = torch.where(sg == 1, -v, v)
            m = torch.nonzero((ds == 4) & (do == 0))[:, 0]
            if len(m):
                R, C = r[m], c[m]
                x, y = self.s[sp][R], self.s[sp][C]
                cre, des = x & ~y, y & ~x
                o, i = _low(cre), _low(des)
                q, j = _low(cre & (cre - 1)), _low(des & (des - 1))
                v = self.eri[o, i, q, j] - self.eri[o, j, q, i]
                st = [self.s[0][C], self.s[1][C]]
                sg = self._sign(*st, 2 * i + sp, 2 * o + sp)
                one = torch.ones_like(i)
                st[sp] = st[sp] ^ (one << i) ^ (one << o)
                sg = sg + self._sign(*st, 2 * j + sp, 2 * q + sp)
                out[m] = torch.where((sg & 1) == 1, -v, v)
        m = torch.nonzero((da == 2) & (db == 2))[:, 0]
        if len(m):
            R, C = r[m], c[m]
            a, b, x, y = self.s[0][C], self.s[1][C], self.s[0][R], self.s[1][R]
            o, i, q, j = _low(x & ~a), _low(a & ~x), _low(y & ~b), _low(b & ~y)
            one = torch.ones_like(i)
            sg = self._sign(a, b, 2 * i, 2 * o) + self._sign(a ^ (one << i) ^ (one << o), b, 2 * j + 1, 2 * q + 1)
            v = self.eri[o, i, q, j]
            out[m] = torch.where((sg & 1) == 1, -v, v)
        return out

    def pairs(self):
        """The connected pairs, a block of rows at a time: row, column, element."""
        st, inv, dist = [], [], []
        for v in self.s:
            u, at = torch.unique(v, return_inverse=True)
            st.append(u)
            inv.append(at)
            d = torch.empty(len(u), len(u), dtype=torch.uint8, device="cuda")
            for b in range(0, len(u), 2048):
                d[b:b + 2048] = _pop(u[b:b + 2048, None] ^ u).to(torch.uint8)
            dist.append(d)
        step = max(1, min(4096, 400_000_000 // self.N))
        for b in range(0, self.N, step):
            da = dist[0][inv[0][b:b + step]].index_select(1, inv[0])
            db = dist[1][inv[1][b:b + step]].index_select(1, inv[1])
            tot = da + db
            for at in torch.nonzero((tot > 0) & (tot <= 4)).split(20_000_000):
                r, c = at[:, 0], at[:, 1]
                x, y = da[r, c].long(), db[r, c].long()
                yield r + b, c, self.elements(r + b, c, x, y)

    def sigma(self, x):
        """H x for the columns of x (N, k)."""
        y = self.diag[:, None] * x
        for r, c, v in self.pairs():
            y.index_add_(0, r, v[:, None] * x[c])
        return y

    def lowest(self, k):
        """The lowest eigenvalues seen by a Krylov space from the first unit vector (one root)."""
        r, c, v = (torch.cat(t) for t in zip(*self.pairs()))
        H = torch.sparse_coo_tensor(torch.stack([r, c]), v, (self.N, self.N)).coalesce().to_sparse_csr()
        q = torch.zeros(self.N, dtype=torch.float64, device="cuda")
        q[0] = 1.0
        Q, al, be = [q], [], []
        for _ in range(min(self.N - 1, 200)):
            w = self.diag * Q[-1] + torch.mv(H, Q[-1])
            al.append(float(w @ Q[-1]))
            B = torch.stack(Q)
            for _ in range(2):
                w = w - B.T @ (B @ w)
            be.append(float(w.norm()))
            if be[-1] < 1e-10:
                break
            Q.append(w / be[-1])
        T = np.diag(al) + np.diag(be[:len(al) - 1], 1) + np.diag(be[:len(al) - 1], -1)
        return np.linalg.eigvalsh(T)[:k]

    def rdm(self, c):
        """Spatial 2-RDM [p, q, r, s] = sum <a+_p a+_q a_s a_r> over the spins of p = r and q = s, and 1-RDM."""
        n, m = self.n, 2 * self.n
        low = [torch.zeros(self.N, dtype=torch.int64, device="cuda"), None]
        idx, row, val = [], [], []
        one = torch.ones((), dtype=torch.int64, device="cuda")
        key = lambda a, b: torch.stack([a, b], 1)  # noqa: E731
        for P in range(m):
            for Q in range(P):
                sel = torch.nonzero((self.occ[P & 1][:, P >> 1] > 0) & (self.occ[Q & 1][:, Q >> 1] > 0))[:, 0]
                a, b = self.s[0][sel], self.s[1][sel]
                p, q = (torch.full_like(a, t) for t in (P, Q))
                sg = self._below(a, b, p) + self._below(a, b, q) - 1  # a_Q a_P, P > Q
                a, b = [t ^ ((one << (P >> 1)) if P & 1 == s else 0) ^ ((one << (Q >> 1)) if Q & 1 == s else 0)
                        for s, t in ((0, a), (1, b))]
                idx.append(key(a, b))
                row.append(torch.full_like(sel, P * (P - 1) // 2 + Q))
                val.append(torch.where((sg & 1) == 1, -c[sel], c[sel]))
        keys, at = torch.unique(torch.cat(idx), dim=0, return_inverse=True)
        row, val = torch.cat(row), torch.cat(val)
        order = torch.argsort(at)
        at, row, val = at[order], row[order], val[order]
        npair = m * (m - 1) // 2
        G = torch.zeros(npair, npair, dtype=torch.float64, device="cuda")
        step = 100_000
        cut = torch.searchsorted(at, torch.arange(0, len(keys) + step, step, device="cuda")).tolist()
        for k, (b, f) in enumerate(zip(cut, cut[1:])):
            M = torch.zeros(npair, step, dtype=torch.float64, device="cuda")
            M[row[b:f], at[b:f] - k * step] = val[b:f]
            G += M @ M.T
        # G[PQ, RS] = <a+_P a+_Q a_S a_R>; summed over spins onto the spatial indices
        four = torch.zeros(m, m, m, m, dtype=torch.float64, device="cuda")
        P, Q = torch.tril_indices(m, m, -1, device="cuda")
        for (x, y, s1) in ((P, Q, 1.0), (Q, P, -1.0)):
            for (z, w, s2) in ((P, Q, 1.0), (Q, P, -1.0)):
                four[x[:, None], y[:, None], z[None], w[None]] = s1 * s2 * G
        two = torch.zeros(n, n, n, n, dtype=torch.float64, device="cuda")
        for s in (0, 1):
            for t in (0, 1):
                two += four[s::2, t::2, s::2, t::2]
        ne = float(self.occ[0][0].sum() + self.occ[1][0].sum())
        return two, torch.einsum("pqrq->pr", two) / (ne - 1.0)


def exact(case, seed):
    """What run() returns in plain FP64. None: whole runs and eigenvectors (defined up to the solver's
    tolerance), perturbation sums (thousands of millions of candidate determinants in plain torch, or drawn by the
    engine's own sampler) and spaces whose pairs take too long to look through."""
    kind, n = case["kind"], case["norb"]
    if kind not in ("sigma", "grow", "davidson", "rdm") or case["ndets"] > 420000:
        return None
    if kind == "rdm" and case["ndets"] * case["na"] * case["nb"] > 4e5:
        return None
    if kind == "davidson" and (case["roots"] > 1 or case["ndets"] > 90000):
        return None
    s = prepare(case, seed)
    if kind == "sigma":
        ex = _Exact(s["dets"], n)
        x = s["x"]
        if case["call"] == "host":
            x = torch.from_numpy(x).cuda()
        elif case["call"] == "packed":
            x = x[:, :case["k"]].T.double()
        y = ex.sigma(x.T.contiguous()).T.contiguous()
        return y.cpu().numpy() if case["call"] == "host" else y
    if kind == "grow":
        e = s["e"]
        e.set_dets(s["small"])
        e.select(s["cmax"], s["eps"])
        y = _Exact(e.dets(), n).sigma(s["x"].T.contiguous()).T.contiguous()
        return {"nnz": None, "dets": None, "y": y}
    ex = _Exact(s["dets"], n)
    if kind == "davidson":
        return {"E": ex.lowest(1), "x": None, "iterations": None}
    two, one = ex.rdm(torch.from_numpy(s["c"]).cuda())
    return {"two": two.cpu().numpy(), "one": one.cpu().numpy()}
