"""Davidson where a correction lies in the span of the basis."""
import numpy as np
import pytest

from dice_gb300 import engine as eng
from dice_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [True, False])
def test_exhausted_block_of_large_energies(tmp_path, graphs):
    """One electron in 8 orbitals: H is the one-electron matrix, with an uncoupled energy A and a 2 x 2 block of
    eigenvalues A and 3 A; nothing couples them to the rest. The start vector lies in these three, so three vectors
    exhaust them. The Ritz value A then meets the diagonal A to the last digit in some of the starts, and the
    correction is a residual of rounding errors over 1e-12: a long vector in the span of the basis, of which only
    the rounding of its projection is left. That must not be taken for a direction of its own."""
    e = eng.Engine(0)
    e.set_davidson_graphs(graphs)
    n = 8
    dets = np.array([(1 << (2 * k), 0) for k in range(n)], dtype=np.uint64)
    for power in (48, 52, 56, 60):
        for seed in range(64):
            rng = np.random.default_rng(seed)
            A = float(np.round(2.0 ** power * rng.uniform(1, 2)))
            h = np.diag([A, 2 * A, 2 * A] + [5 * A] * (n - 3))
            h[1, 2] = h[2, 1] = A
            path = str(tmp_path / "F")
            synthetic.write_fcidump(path, h, np.zeros((n,) * 4), 1, ms2=1)
            e.read_fcidump(path)
            e.set_dets(dets)
            e.ham_build("fp64")
            x0 = np.zeros((1, n))
            x0[0, :3] = rng.standard_normal(3)
            E, x, _ = e.davidson(x0, tol=1e-7)
            # a 3 x 3 eigenproblem of norm 3 A: some tens of roundings of it
            assert abs(E[0] - A) <= 256 * 2.0 ** -53 * A, (power, seed, A, E)
            assert abs(np.linalg.norm(x) - 1.0) <= 1e-12, (power, seed)
    e.close()
