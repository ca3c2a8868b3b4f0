"""QEq within a scratch budget that holds no more than its k-sum as a library product took: the Gram works block
by block, and the results have the bits of an ample budget."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cell(n, n_grid, seed):
    rng = np.random.default_rng(seed)
    box = np.array([[18.0, 0.0, 0.0], [1.5, 19.0, 0.0], [-1.0, 2.0, 20.0]])
    return box / np.array(n_grid)[:, None], rng.random((n, 3)) @ box, rng


@pytest.mark.parametrize("n", [40, 300, 900])
def test_qeq_in_a_tight_budget(n):
    from pyrepeat_gb300.fit import Context
    n_grid = (20, 22, 24)
    axis, atoms, rng = _cell(n, n_grid, n)
    chi, js = rng.normal(0.2, 0.05, size=n), 0.4 + rng.random(n)
    K = 754  # wave vectors at KMAX 7
    budget = 32 * n * K + 16 * n * n + 16 * (n + 1) ** 2 + (3 << 20)
    out = []
    for hbm in (0, budget):
        q, J, _ = Context(0, hbm_budget=hbm).qeq(n_grid, axis, atoms, chi, js, 0.0, 20.0, 7, want_J=True)
        out.append((q, J))
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][0], out[1][0])
