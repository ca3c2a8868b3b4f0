"""The FP64 normal equations (separable reciprocal sum, tabulated real-space term, exact two-word Gram)
against the oracle's direct sums, over the cutoffs and KMAX that change the term's table, the
k-set and the image counts, and for one and two atoms.  A is a sum of up to 2e4 products of centred
Phi values that both sides form in FP64 (relative rounding below 1e-14 of max |Phi| each), so the
two agree to 1e-11 of the largest entry."""
import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_atoms,kmax,cutoff", [(40, 7, 20.0), (40, 12, 20.0), (40, 3, 9.0), (33, 7, 31.0), (2, 7, 20.0),
                                                 (1, 1, 20.0), (17, 2, 4.0)])
def test_fp64_normal_equations(n_atoms, kmax, cutoff, gpu_ctx, oracle_mod):
    import torch
    from pyrepeat_gb300 import _lib
    cube, _ = load_golden("tricmini")
    cube.atom_pos, cube.atom_index = cube.atom_pos[:n_atoms], cube.atom_index[:n_atoms]
    cube.symm_groups, cube.resp, cube.kmax, cube.cutoff = None, None, kmax, cutoff
    of = oracle_mod.OracleFit(cube)
    A, b, _, _ = of.normal_equations()
    kept = torch.from_numpy(np.ascontiguousarray(of.kept, dtype=np.int32)).cuda()
    V = torch.from_numpy(np.ascontiguousarray(of.Vc, dtype=np.float64)).cuda()
    ew = gpu_ctx.ewald(cube.n_grid, cube.axis_vector, cutoff, kmax)
    try:
        Ag, bg, _ = gpu_ctx.gram(ew, cube.atom_pos, kept, V, _lib.PREC_FP64)
    finally:
        ew.close()
    assert np.abs(Ag.cpu().numpy() - A).max() <= 1e-11 * np.abs(A).max()
    assert np.abs(bg.cpu().numpy() - b).max() <= 1e-11 * max(np.abs(b).max(), np.abs(A).max())
