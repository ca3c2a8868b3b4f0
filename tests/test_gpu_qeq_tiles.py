"""The QEq Coulomb matrix at the pair kernel's tile edges, with image lists longer than one 32-shift
chunk, atoms nearer than the term's table begins, and a left-handed cell (whose k-space weights are
negative), against the oracle's matrix within the 1e-12 of the other QEq tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kmax,cutoff,left", [(1, 7, 20.0, False), (31, 7, 20.0, False), (32, 0, 20.0, False),
                                                (33, 3, 31.0, False), (65, 7, 9.0, True), (97, 7, 20.0, True)])
def test_coulomb_matrix(n, kmax, cutoff, left, gpu_ctx, oracle_mod):
    rng = np.random.default_rng(n)
    ng = np.array([20, 22, 24])
    box = np.array([[15.0, 0.0, 0.0], [1.5, 16.0, 0.0], [-1.0, 2.0, 17.0]])
    if left:
        box = box[[1, 0, 2]]
    atoms = rng.random((n, 3)) @ box
    if n > 2:
        atoms[1] = atoms[0] + 0.1  # closer than half a Bohr
    js = 0.4 + rng.random(n)
    _, J, _ = gpu_ctx.qeq(ng, box / ng[:, None], atoms, np.zeros(n), js, 0.0, cutoff, kmax, want_J=True)
    ref = oracle_mod.qeq_matrix(atoms, box, cutoff, kmax, js)
    assert np.array_equal(J, J.T)
    assert np.abs(J - ref).max() <= 1e-12 * np.abs(ref).max()
