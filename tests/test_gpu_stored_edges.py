"""The Hamiltonian's build and its products at the sizes where their kernels
change path: rows of one piece and of many, rows past the shared-memory merge,
short rows (several to a warp), strings of 32 bits and of more, a beta group
with more partners than its buffer holds, and spaces at a sort tile's edge.
FP64 elements equal the oracle's bit for bit; products lie within the rounding of
their sums."""
import itertools

import numpy as np
import pytest

from dice_gb300 import engine as eng
from dice_gb300 import synthetic
from dice_gb300.shard import ref_order
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

U64, U32 = 2.0 ** -53, 2.0 ** -24


@pytest.fixture(scope="module")
def system(tmp_path_factory):
    made = {}

    def get(norb, nelec):
        if (norb, nelec) not in made:
            d = tmp_path_factory.mktemp("s%d_%d" % (norb, nelec))
            h, eri = synthetic.molecular_integrals(norb, 8, 100 + norb)
            # the file's integrals cut at 1e-6 of the largest: a few lines fewer, the same path
            synthetic.write_fcidump(str(d / "FCIDUMP"), h, eri, nelec, ms2=nelec % 2, tol=1e-6)
            e = eng.Engine(0)
            e.read_fcidump(str(d / "FCIDUMP"))
            made[norb, nelec] = e, orc.Oracle(str(d / "FCIDUMP"))
        return made[norb, nelec]

    yield get
    for e, _ in made.values():
        e.close()


def _words(a, b):
    """(word 0, word 1) of the strings a, b: alpha on even bits, beta on odd."""
    w = sum(1 << (2 * k) for k in range(64) if a >> k & 1) | sum(2 << (2 * k) for k in range(64) if b >> k & 1)
    return w & (2 ** 64 - 1), w >> 64


def _star(norb, na, nb, n, seed):
    """The lowest determinant and n - 1 others one or two electrons from it, in random order."""
    rng = np.random.default_rng(seed)
    a0, b0 = (1 << na) - 1, (1 << nb) - 1

    def moved(s, ne, times):
        times = min(times, ne, norb - ne)
        occ = rng.choice(ne, times, replace=False)
        emp = ne + rng.choice(norb - ne, times, replace=False)
        for o, v in zip(occ, emp):
            s ^= 1 << int(o) | 1 << int(v)
        return s

    out = {(a0, b0): None}
    while len(out) < n:
        ta, tb = ((0, 1), (1, 0), (1, 1), (1, 1), (1, 1), (2, 0), (0, 2))[rng.integers(7)]
        out[moved(a0, na, ta), moved(b0, nb, tb)] = None
    d = np.array([_words(a, b) for a, b in out], dtype=np.uint64)
    return d[rng.permutation(len(d))]


def _lower(n, rp, col, val):
    """Off-diagonal entries below the diagonal, by (row, column)."""
    row = np.repeat(np.arange(n, dtype=np.int64), np.diff(rp))
    m = col < row
    o = np.lexsort((col[m], row[m]))
    return row[m][o], col[m][o].astype(np.int64), val[m][o]


def _check(e, o, dets, modes=("fp64", "mixed"), ks=(1, 2, 3, 4)):
    n = len(dets)
    rng = np.random.default_rng(n)
    X = rng.standard_normal((4, n))
    oref = _lower(n, *o.ham(dets))
    ref = np.stack([o.sigma(x) for x in X])
    e.set_dets(dets)
    diag = e.diag()
    assert np.array_equal(diag, [o.energy(d) for d in dets])
    longest = 0
    for mode in modes:
        nnz = e.ham_build(mode)
        rp, col, val = e.ham_export(nnz)
        longest = int(np.diff(rp).max())
        got = _lower(n, rp, col, val)
        assert nnz == 2 * len(oref[0])
        assert np.array_equal(got[0], oref[0]) and np.array_equal(got[1], oref[1]), mode
        if mode == "fp64":
            assert np.array_equal(got[2], oref[2])
        else:  # stored as an FP32 head and tail
            assert np.all(np.abs(got[2] - oref[2]) <= 2.0 ** -48 * np.abs(oref[2]))
        row = np.repeat(np.arange(n), np.diff(rp))
        A = np.abs(diag) * np.abs(X)  # |H| |x|, and its rows' lengths: the bound of a sum's rounding
        for j in range(4):
            A[j] += np.bincount(row, np.abs(val) * np.abs(X[j][col]), n)
        f64 = 2 * (np.diff(rp) + 4) * U64 * A  # the oracle's sum and the engine's
        for k in ks:
            if mode == "fp64":
                for m in ("fp64", "direct"):
                    assert np.all(np.abs(e.sigma(X[:k], m) - ref[:k]) <= f64[:k]), (m, k)
            else:
                # value, x, product and result rounded to FP32; the sums compensated
                f32 = 6 * U32 * A
                assert np.all(np.abs(e.sigma(X[:k], "mixed") - ref[:k]) <= f32[:k]), k
                # head and tail of the values and of x: 2^-48 each
                assert np.all(np.abs(e.sigma(X[:k], "fp64") - ref[:k]) <= f64[:k] + 64 * 2.0 ** -48 * A[:k]), k
    return longest


# the lowest determinant's row holds n - 1 entries: one piece of the FP64 walk (2,048), of the FP32 walk
# (4,096), the merges in shared memory (2,560 and 7,168) and a sort tile (4,096), each to the entry, and several
# pieces
@pytest.mark.parametrize("n", [2049, 2050, 2561, 2562, 3073, 3074, 4096, 4097, 4098, 7169, 7170, 8194])
def test_long_rows(system, n):
    e, o = system(20, 20)
    assert _check(e, o, _star(20, 10, 10, n, n)) == n - 1


# strings of 32 bits and of 33, odd electrons, the widest; short rows beside one long one
@pytest.mark.parametrize("norb,na,nb,n", [(32, 8, 7, 700), (33, 8, 7, 700), (33, 16, 16, 5000), (64, 20, 20, 900),
                                          (64, 3, 2, 33), (2, 1, 1, 2)])
def test_string_widths_and_short_rows(system, norb, na, nb, n):
    e, o = system(norb, na + nb)
    _check(e, o, _star(norb, na, nb, n, norb + n))


@pytest.mark.parametrize("alphas", [1, 3])
def test_beta_group_larger_than_its_buffer(system, alphas):
    """All 1,716 beta strings of 6 electrons in 13 orbitals on the same alpha string: 357 partners each."""
    e, o = system(13, 12)
    bs = [sum(1 << k for k in c) for c in itertools.combinations(range(13), 6)]
    al = [0b111111, 0b1011111, 0b1111110000000][:alphas]
    dets = np.array([_words(a, b) for a in al for b in bs], dtype=np.uint64)
    assert _check(e, o, dets[np.random.default_rng(0).permutation(len(dets))]) >= 357


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("norb,n", [(20, 3000), (33, 1200)])
def test_appended_space_equals_full_build(system, norb, n, mode):
    """Fewer new determinants than old ones extend the stored rows, as many or more rebuild them: one to
    either side of the line, one new determinant and none."""
    e, _ = system(norb, 20)
    dets = _star(norb, 10, 10, n, 7)
    for old in (n // 2 - 1, n // 2, n // 2 + 1, n - 1, n):
        tail = dets[old:][ref_order(dets[old:])]
        e.set_dets(np.concatenate([dets[:old], tail]))
        full = e.ham_export(e.ham_build(mode))
        e.set_dets(dets[:old])
        e.ham_build(mode)
        if len(tail):
            e.append_dets(tail)
        got = e.ham_export(e.ham_build(mode))
        for a, b in zip(got, full):
            assert np.array_equal(a, b), old


# 8,192 entries of x pass through pinned memory, one more goes by the copy engine
@pytest.mark.parametrize("n,k", [(1, 1), (4096, 2), (4097, 2), (8192, 1), (8193, 1), (2730, 3), (2731, 3), (2048, 4)])
def test_host_vectors_equal_device_vectors(system, n, k):
    import torch
    e, _ = system(20, 20)
    e.set_dets(_star(20, 10, 10, n, 3))
    x = np.random.default_rng(n).standard_normal((k, n))
    for build, modes in (("fp64", ("fp64", "direct", "direct_mixed")), ("mixed", ("mixed", "fp64"))):
        e.ham_build(build)
        for mode in modes:
            xd = torch.tensor(x, device="cuda")
            yd = torch.full_like(xd, float("nan"))
            torch.cuda.synchronize()
            e.sigma_device(xd.data_ptr(), yd.data_ptr(), k, n, mode=mode)
            torch.cuda.synchronize()
            assert np.array_equal(e.sigma(x, mode), yd.cpu().numpy()), (build, mode)


@pytest.mark.parametrize("norb", [32, 33, 50])
def test_selection_and_pt_by_string_width(system, norb):
    e, o = system(norb, 13)
    dets = _star(norb, 7, 6, 60, norb)
    c = np.random.default_rng(norb).standard_normal(60) * 0.2
    c[0] = 0.9
    e.set_selection_params()
    e.set_dets(dets)
    got, ref = e.select_candidates(np.abs(c), 1e-4), o.select(dets, np.abs(c), 1e-4, dets[ref_order(dets)])
    assert len(got) > 100 and np.array_equal(got, ref)
    E0 = float(e.diag().min()) - 30.0
    e2 = e.pt_deterministic(c, E0, 1e-5)
    ref, st = o.pt_det(dets, c, E0, 1e-5)
    got = e.pt_stats()
    assert (got["candidates"], got["unique"]) == (st["outside"], st["unique"])
    assert abs(e2 - ref) <= 1e-10 * abs(ref)


@pytest.mark.parametrize("norb,na,nb,n", [(20, 10, 10, 4098), (33, 8, 7, 700), (64, 3, 2, 33), (2, 1, 1, 2)])
def test_density_matrices_by_string_width(system, norb, na, nb, n):
    e, o = system(norb, na + nb)
    dets = _star(norb, na, nb, n, norb + n)
    c = np.random.default_rng(n).standard_normal(n)
    c /= np.linalg.norm(c)
    e.set_dets(dets)
    s2, s1 = e.rdm(ci=c)
    r2, r1 = o.rdm(dets, c)
    # sums of the order of n terms, whose absolute values add up to at most (electrons)^2
    tol = 4 * (n + 16) * U64 * (na + nb) ** 2
    assert np.max(np.abs(s2 - r2)) <= tol and np.max(np.abs(s1 - r1)) <= tol
