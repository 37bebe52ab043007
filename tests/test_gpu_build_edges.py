"""The Hamiltonian build on lists of determinants at the edge of what the calls
take: determinants given more than once, spaces that have not changed, builds that
run out of memory half way."""
import itertools

import numpy as np
import pytest
from scipy import sparse

from dice_gb300 import engine as eng
from dice_gb300.shard import ref_order
from test_gpu_stored_edges import U64, _lower, _star, _words, system  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


def _grouped(alphas):
    """All 1,716 beta strings of 6 electrons in 13 orbitals on each alpha string: groups that are looked up in the
    index (more than 48 determinants)."""
    bs = [sum(1 << k for k in c) for c in itertools.combinations(range(13), 6)]
    return np.array([_words(a, b) for a in alphas for b in bs], dtype=np.uint64)


def _expanded(o, dets):
    """Lower triangle of the list's matrix: that of its distinct determinants, copied (two copies of one
    determinant are not connected)."""
    u, at = np.unique(dets, axis=0, return_inverse=True)
    at = at.reshape(-1)
    r, c, v = _lower(len(u), *o.ham(u))
    # entries by their place, so that elements of exactly zero stay entries
    k = np.arange(1, len(r) + 1, dtype=np.float64)
    H = sparse.coo_matrix((np.r_[k, k], (np.r_[r, c], np.r_[c, r])), shape=(len(u),) * 2).tocsr()
    H = sparse.tril(H[at][:, at], -1).tocoo()
    s = np.lexsort((H.col, H.row))
    return H.row[s].astype(np.int64), H.col[s].astype(np.int64), v[H.data[s].astype(np.int64) - 1]


# copies of a few determinants, of the lowest one, and more than 64 of one (a run of the index longer than a
# slot's length field)
@pytest.mark.parametrize("copies", [(1,), (2, 1, 1, 3), (70,)])
@pytest.mark.parametrize("norb", [13, 33])
def test_repeated_determinants(system, norb, copies):  # noqa: F811
    e, o = system(norb, 12)
    dets = _grouped([0b111111, 0b1011111, 0b1101111])
    rng = np.random.default_rng(len(copies))
    twice = np.concatenate([[0], rng.choice(np.arange(1, len(dets)), len(copies) - 1, replace=False)])
    dets = np.concatenate([dets] + [np.repeat(dets[i:i + 1], m, 0) for i, m in zip(twice, copies)])
    dets = dets[rng.permutation(len(dets))]
    n = len(dets)
    ref = _expanded(o, dets)
    x = rng.standard_normal(n)
    for mode in ("fp64", "mixed"):
        e.set_dets(dets)
        nnz = e.ham_build(mode)
        assert nnz == 2 * len(ref[0])
        rp, col, val = e.ham_export(nnz)
        got = _lower(n, rp, col, val)
        assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1]), mode
        assert np.all(np.abs(got[2] - ref[2]) <= (0.0 if mode == "fp64" else 2.0 ** -48) * np.abs(ref[2]))
        if mode == "fp64":
            diag = e.diag()
            row = np.repeat(np.arange(n), np.diff(rp))
            y = diag * x + np.bincount(row, val * x[col], n)
            A = np.abs(diag * x) + np.bincount(row, np.abs(val * x[col]), n)
            for m in ("fp64", "direct"):
                assert np.all(np.abs(e.sigma(x, m) - y) <= 2 * (np.diff(rp) + 4) * U64 * A), m
        # the same list reached by extending stored rows
        tail = np.unique(dets, axis=0)
        tail = tail[ref_order(tail)][-40:]
        old = np.array([d for d in dets if not (tail == d).all(1).any()], dtype=np.uint64)
        e.set_dets(np.concatenate([old, tail]))
        full = e.ham_export(e.ham_build(mode))
        e.set_dets(old)
        e.ham_build(mode)
        e.append_dets(tail)
        for a, b in zip(e.ham_export(e.ham_build(mode)), full):
            assert np.array_equal(a, b), mode


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_unchanged_space_is_not_built_again(system, mode):  # noqa: F811
    """A repeated build of the same space keeps the stored rows: nothing is launched but the mixed form's compact
    copy (lengths, their scan, the copy)."""
    e, _ = system(20, 20)
    e.set_dets(_star(20, 10, 10, 3000, 5))
    nnz = e.ham_build(mode)
    first = e.ham_export(nnz)
    before = e.launch_count()
    assert e.ham_build(mode) == nnz
    assert e.launch_count() - before <= (0 if mode == "fp64" else 5)
    for a, b in zip(e.ham_export(nnz), first):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("build", ["fp64", "rows", "grown"])
def test_build_that_runs_out_of_memory(system, build):  # noqa: F811
    """Wherever a build stops for want of memory, the matrix that was there is either still there or refused,
    and the next build is complete."""
    e, _ = system(20, 20)
    dets = _star(20, 10, 10, 4000, 11)
    tail = dets[1500:][ref_order(dets[1500:])]
    full = np.concatenate([dets[:1500], tail])
    rng = np.random.default_rng(1)
    x, xf = rng.standard_normal(1500 if build == "grown" else 4000), rng.standard_normal(4000)

    def prepare():
        e.set_dets(full[:1500] if build == "grown" else full)
        e.ham_build("mixed")

    def attempt():
        if build == "grown":
            e.append_dets(tail)
            return e.ham_build("mixed")
        return e.ham_build("fp64") if build == "fp64" else e.ham_build_rows(100, 3900, "mixed")

    prepare()
    y = e.sigma(x, "mixed")
    e.set_dets(full)
    nnz = e.ham_build("mixed")
    yf = e.sigma(xf, "mixed")
    refused = held = 0
    cap, step = 2.0 ** 20, 2.0
    while True:  # the smallest sufficient cap from below, then in small steps
        prepare()
        e.set_alloc_cap(int(cap))
        try:
            attempt()
            ok = True
        except eng.ShciError as err:
            assert err.code == 4
            ok = False
        finally:
            e.set_alloc_cap(0)
        if ok:
            if step < 1.01:
                break
            cap, step = cap / step, 1.0 + (step - 1.0) / 8.0  # back to the last cap that was too small
            continue
        if e.ndets() == len(x):
            try:
                assert np.array_equal(e.sigma(x, "mixed"), y)
                held += 1
            except eng.ShciError as err:
                assert err.code == 7
                refused += 1
        if build == "grown":
            try:
                e.append_dets(tail)  # the append itself may have been what failed
            except eng.ShciError as err:
                assert err.code == 1
        assert e.ham_build("mixed") == nnz
        assert np.array_equal(e.sigma(xf, "mixed"), yf)
        cap *= step
    assert build == "grown" or refused > 0


@pytest.mark.parametrize("norb", [20, 32, 33, 64])
def test_appended_determinants_lie_within_the_orbitals(system, norb):  # noqa: F811
    """An electron past the last orbital, or one electron too many, is refused and the space stays as it was."""
    e, _ = system(norb, 6)
    dets = _star(norb, 3, 3, 20, 2)
    e.set_dets(dets)
    beyond = [(1 << (2 * norb)) | 0b11111] if norb < 64 else []
    for w in beyond + [(1 << (2 * norb - 1)) | 0b111111]:
        with pytest.raises(eng.ShciError) as err:
            e.append_dets(np.array([(w & (2 ** 64 - 1), w >> 64)], dtype=np.uint64))
        assert err.value.code == 1
    w = (3 << (2 * norb - 2)) | (15 << (2 * norb - 6))  # the last three orbitals, doubly occupied
    e.append_dets(np.array([(w & (2 ** 64 - 1), w >> 64)], dtype=np.uint64))
    assert np.array_equal(e.dets(), np.concatenate([dets, [[w & (2 ** 64 - 1), w >> 64]]]))


@pytest.mark.parametrize("mode", ["fp64", "mixed", "direct"])
def test_refused_space_leaves_the_old_one(system, mode):  # noqa: F811
    """A list with a wrong determinant is refused; the space and its matrix are still there."""
    e, _ = system(20, 20)
    dets = _star(20, 10, 10, 300, 4)
    e.set_dets(dets)
    e.ham_build(mode)
    x = np.random.default_rng(0).standard_normal(300)
    y = e.sigma(x, mode)
    e.sigma(x + 1.0, mode)  # y is no longer in the context's buffers
    bad = dets[:200].copy()
    bad[150, 0] ^= np.uint64(1)  # an electron too few or too many
    with pytest.raises(eng.ShciError) as err:
        e.set_dets(bad)
    assert err.value.code == 1
    assert np.array_equal(e.dets(), dets) and np.array_equal(e.sigma(x, mode), y)


def test_no_room_for_the_compact_copy(system):  # noqa: F811
    """A mixed build whose compact copy finds no memory keeps its int32 columns, says so in the bytes of a sigma, and
    gives the same products."""
    e, _ = system(20, 20)
    n = 4000
    e.set_dets(_star(20, 10, 10, n, 12))
    nnz = e.ham_build("mixed")
    rp, col, val = e.ham_export(nnz)
    x = np.random.default_rng(2).standard_normal(n)
    y, small = e.sigma(x, "mixed"), e.sigma_bytes("mixed", 1)

    e.set_alloc_cap(1)  # the unchanged space: only the copy is made again
    try:
        assert e.ham_build("mixed") == nnz
    finally:
        e.set_alloc_cap(0)
    assert e.sigma_bytes("mixed", 1) > small
    # compensated sums of the same products in another order: 2^-40 of their absolute values
    A = np.bincount(np.repeat(np.arange(n), np.diff(rp)), np.abs(val * x[col]), n) + np.abs(e.diag() * x)
    assert np.all(np.abs(e.sigma(x, "mixed") - y) <= 2.0 ** -40 * A)
