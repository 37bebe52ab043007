"""Sorts take the digits in which their keys differ: a frozen core and empty
upper orbitals cost no passes, and the order is the same wherever the differing
bits lie (within a word, across both, at a word's sign bit)."""
import itertools

import numpy as np
import pytest

from dice_gb300.shard import ref_order
from test_gpu_stored_edges import _check, _words, system  # noqa: F401  (fixture)
from test_gpu_units import _dets, mol24  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


def _window(lo, n, na, nb, keep, seed):
    """Determinants with all orbitals below lo doubly occupied and na + nb electrons in the n orbitals from lo."""
    core = (1 << lo) - 1
    al, be = ([core | sum(1 << (lo + k) for k in c) for c in itertools.combinations(range(n), m)] for m in (na, nb))
    d = np.array([_words(a, b) for a in al for b in be], dtype=np.uint64)
    return d[np.random.default_rng(seed).permutation(len(d))[:keep]]


# 6 orbitals (12 bits: two digits) low, about the middle of a word, and across the words' border (spin orbitals 58 to
# 69, bits 58 to 63 and 0 to 5); the highest (116 to 127)
@pytest.mark.parametrize("lo", [0, 17, 29, 58])
def test_window_of_64_orbitals(system, lo):  # noqa: F811
    e, o = system(64, 2 * lo + 6)
    dets = _window(lo, 6, 3, 3, 60, lo)
    c = np.abs(np.random.default_rng(lo).standard_normal(len(dets)))
    e.set_selection_params(lo, 6)
    e.set_dets(dets)
    n0 = e.launch_count()
    got = e.select_candidates(c, 1e-5)
    n1 = e.launch_count()
    e.set_selection_params()
    ref = o.select(dets, c, 1e-5, dets[ref_order(dets)], ncore=lo, nact=6)
    assert len(got) > 50 and np.array_equal(got, ref)
    # two digits of at most four launches, and the hash, the slices, the walk, the split, the join and the unique pass
    assert n1 - n0 <= 2 * 4 + 14
    n0 = e.launch_count()
    e.ham_build("fp64")
    # alpha and beta strings one digit each, beta strings again one, partial strings what lo + 6 orbitals take, groups
    # one; 30 launches for the tables, the rows and the diagonal
    assert e.launch_count() - n0 <= (4 + (lo + 13) // 8) * 4 + 30
    _check(e, o, dets, ks=(1,))


def test_space_grown_from_one_determinant(system):  # noqa: F811
    """The differing bits grow with the space: selections and appends give what the same list given whole gives."""
    e, _ = system(64, 12)
    e.set_selection_params()
    start = np.array([_words(0b111111, 0b111111)], dtype=np.uint64)
    e.set_dets(start)
    e.ham_build("fp64")
    e.select(np.ones(1), 2e-2)
    e.ham_build("fp64")
    high = np.array([_words(0b11111 | 1 << 63, 0b11111 | 1 << 63), _words(0b11111 | 1 << 40, 0b111111)], dtype=np.uint64)
    high = np.array([d for d in high[ref_order(high)] if not (e.dets() == d).all(1).any()], dtype=np.uint64)
    assert len(high) > 0
    e.append_dets(high)
    grown = e.dets()
    rows = e.ham_export(e.ham_build("fp64"))
    c = np.random.default_rng(0).uniform(0.1, 1.0, len(grown))
    cand = e.select_candidates(c, 1e-2)
    e2 = e.pt_deterministic(c, float(e.diag().min()) - 30.0, 1e-3)
    st = e.pt_stats()
    e.set_dets(grown)
    for a, b in zip(rows, e.ham_export(e.ham_build("fp64"))):
        assert np.array_equal(a, b)
    assert len(cand) > 100 and np.array_equal(e.select_candidates(c, 1e-2), cand)
    assert e.pt_deterministic(c, float(e.diag().min()) - 30.0, 1e-3) == e2
    assert e.pt_stats()["unique"] == st["unique"] > 100


# 256 counts per tile of 4,096 keys, scanned in chunks of 4,096 counts: up to 256 chunks (16,777,216 keys) in two
# launches, beyond in three. A parent of 12 + 12 electrons in 24 orbitals has 288 + 8,712 + 20,736 = 29,736
# connections: 564 parents stay below, 565 do not.
@pytest.mark.parametrize("n", [564, 565])
def test_scan_at_its_chunk_limit(mol24, n):  # noqa: F811
    e, _ = mol24
    dets = _dets(n, 31)
    c = np.full(n, n ** -0.5)
    e.set_selection_params()
    e.set_dets(dets)
    E0 = float(e.diag().min()) - 30.0
    e2 = e.pt_deterministic(c, E0, 1e-12)
    whole = e.pt_stats()
    assert whole["partitions"] == 1 and (whole["candidates"] <= 16777216) == (n == 564)
    assert abs(whole["candidates"] - 16777216) < 30000
    e.set_pt_batch(whole["candidates"] // 5)
    p2 = e.pt_deterministic(c, E0, 1e-12)
    parts = e.pt_stats()
    e.set_pt_batch(0)
    assert parts["partitions"] > 1
    assert (whole["candidates"], whole["unique"]) == (parts["candidates"], parts["unique"])
    # the same terms, summed in parts: some 1e7 terms of one sign
    assert abs(e2 - p2) <= 1e-11 * abs(e2)
