"""Work units of the selection and of the PT generator: parents cut into
slices (one parent, a few heavy ones, heavy and light ones mixed, more slices
than the unit list holds) give what the oracle, or the parents taken apart,
give."""
import numpy as np
import pytest

from dice_gb300 import engine as eng
from dice_gb300 import synthetic
from dice_gb300.shard import ref_order
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mol24(tmp_path_factory):
    d = tmp_path_factory.mktemp("mol24")
    synthetic.make_workload("mol24", str(d))
    e = eng.Engine(0)
    e.read_fcidump(str(d / "FCIDUMP"))
    yield e, orc.Oracle(str(d / "FCIDUMP"))
    e.close()


def _spread(x):
    return sum(((int(x) >> k) & 1) << (2 * k) for k in range(24))


def _dets(n, seed, orbs=24):
    """n distinct determinants of 12 alpha and 12 beta electrons in the lowest `orbs` orbitals."""
    rng = np.random.default_rng(seed)
    out = {}
    while len(out) < n:
        a, b = (sum(1 << int(o) for o in rng.choice(orbs, 12, replace=False)) for _ in range(2))
        out[_spread(a) | (_spread(b) << 1)] = None
    return np.array([(w, 0) for w in out], dtype=np.uint64)


# the oracle's walk over the lists in Python-call-free C++ takes about a second for 40 heavy parents
@pytest.mark.parametrize("n,light", [(1, 0), (2, 1), (33, 20), (40, 0)])
def test_cut_parents_select_what_the_oracle_selects(mol24, n, light):
    e, o = mol24
    dets = _dets(n, 11 * n)
    c = np.ones(n)
    c[n - light:] = 1e-6  # below every threshold of the lists: whole parents
    e.set_selection_params()
    e.set_dets(dets)
    got = e.select_candidates(c, 1e-5)
    ref = o.select(dets, c, 1e-5, dets[ref_order(dets)])
    assert len(got) == len(ref) > 1000 and np.array_equal(got, ref)


@pytest.mark.parametrize("n,light", [(1, 0), (3, 1), (12, 0)])
def test_cut_parents_give_the_oracles_pt(mol24, n, light):
    e, o = mol24
    dets = _dets(n, 5 + n)
    c = np.full(n, 0.3)
    c[n - light:] = 1e-5
    e.set_selection_params()
    e.set_dets(dets)
    E0 = float(e.diag().min()) - 30.0
    e2 = e.pt_deterministic(c, E0, 1e-5)
    ref, st = o.pt_det(dets, c, E0, 1e-5)
    got = e.pt_stats()
    assert (got["candidates"], got["unique"]) == (st["outside"], st["unique"])
    assert abs(e2 - ref) <= 1e-10 * abs(ref)


def test_more_slices_than_the_list_holds(mol24):
    """15,000 heavy parents claim more slices than the unit list has room for; each quarter of them alone
    does not. The selected determinants are the union of the quarters'."""
    e, _ = mol24
    dets = _dets(15000, 3, orbs=15)
    e.set_selection_params(0, 15)  # few candidates: the list entries are walked all the same
    e.set_dets(dets)
    c = np.ones(len(dets))
    whole = e.select_candidates(c, 1e-7)
    parts = [e.select_candidates(np.where(np.arange(len(dets)) % 4 == k, c, 0.0), 1e-7) for k in range(4)]
    ref = np.unique(np.concatenate(parts), axis=0)
    e.set_selection_params()
    assert len(whole) == len(ref) and np.array_equal(np.unique(whole, axis=0), ref)


@pytest.mark.parametrize("n", [16383, 16384, 30000])
def test_slice_size_follows_the_total(mol24, n):
    """From 16,384 parents on a slice's size goes with the entries of all of them: three quarters of the
    coefficients at zero give smaller slices, and the same determinants."""
    e, _ = mol24
    dets = _dets(n, 4, orbs=15)
    e.set_selection_params(0, 15)
    e.set_dets(dets)
    c = np.ones(n)
    whole = e.select_candidates(c, 1e-7)
    parts = [e.select_candidates(np.where(np.arange(n) % 4 == k, c, 0.0), 1e-7) for k in range(4)]
    ref = np.unique(np.concatenate(parts), axis=0)
    e.set_selection_params()
    assert len(whole) == len(ref) and np.array_equal(np.unique(whole, axis=0), ref)


def test_pt_tables_follow_the_integrals(tmp_path):
    """Two FCIDUMPs of the same size in turn in one context: each correction is the oracle's for its own
    integrals (the generator's tables are made again when integrals are read)."""
    e = eng.Engine(0)
    got, ref = [], []
    for seed in (1, 2, 1):
        path = str(tmp_path / ("F%d" % seed))
        h, eri = synthetic.molecular_integrals(8, 8, seed)
        synthetic.write_fcidump(path, h, eri, 8)
        e.read_fcidump(path)
        dets = np.array([(0b11111111, 0), (0b110111111, 0)], dtype=np.uint64)
        c = np.array([0.9, 0.4])
        e.set_dets(dets)
        E0 = float(e.diag().min()) - 5.0
        got.append(e.pt_deterministic(c, E0, 1e-6))
        ref.append(orc.Oracle(path).pt_det(dets, c, E0, 1e-6)[0])
    e.close()
    assert abs(ref[0] - ref[1]) > 1e-3 * abs(ref[0])
    assert np.allclose(got, ref, rtol=1e-10, atol=0)


# keys per sort: 256 counts per 4,096 keys, scanned in chunks of 4,096; to 256 chunks (16.8 million keys)
# in two launches, beyond in three. Parents of 29,436 connections each (12 + 12 electrons in 24 orbitals).
@pytest.mark.parametrize("n", [2, 3, 570, 600])
def test_sorts_to_either_side_of_a_scans_levels(mol24, n):
    e, _ = mol24
    dets = _dets(n, 31)
    c = np.full(n, n ** -0.5)
    e.set_selection_params()
    e.set_dets(dets)
    E0 = float(e.diag().min()) - 30.0
    e2 = e.pt_deterministic(c, E0, 1e-12)
    whole = e.pt_stats()
    e.set_pt_batch(max(1000, whole["candidates"] // 5))  # parts of a fifth: small sorts
    p2 = e.pt_deterministic(c, E0, 1e-12)
    parts = e.pt_stats()
    e.set_pt_batch(0)
    assert parts["partitions"] > 1
    assert (whole["candidates"], whole["unique"]) == (parts["candidates"], parts["unique"])
    # the same terms, summed in parts: some 1e7 terms of one sign
    assert abs(e2 - p2) <= 1e-11 * abs(e2)
