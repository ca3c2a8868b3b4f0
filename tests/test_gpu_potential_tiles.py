"""rp_potential at tile edges (128 points per CTA, images in rounds of 1536 per CTA, atoms over 32 lanes in
the structure factor), every grid point and chosen ones, against the oracle's Phi q within the 1e-6
of the largest value that the potential is held to."""
import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,npts,kmax,cutoff", [(1, 1, 7, 20.0), (31, 127, 7, 20.0), (33, 129, 3, 20.0), (40, 300, 7, 31.0)])
def test_potential_at_chosen_points(n, npts, kmax, cutoff, gpu_ctx, oracle_mod):
    import torch
    from pyrepeat_gb300 import synth
    cube, g = load_golden("tricmini")
    atoms = np.ascontiguousarray(cube.atom_pos[:n])
    q = np.random.default_rng(n).normal(size=n)
    idx = np.random.default_rng(npts).permutation(np.flatnonzero(g["mask"]))[:npts]
    nx, ny = int(cube.n_grid[0]), int(cube.n_grid[1])
    p = np.stack([idx % nx, (idx // nx) % ny, idx // (nx * ny)], axis=1) @ cube.axis_vector
    box = cube.box_vectors
    _, kv, kc = synth.kspace(box, cutoff, kmax)
    sh = synth.realspace_shifts(box, cutoff)
    zero = int(np.flatnonzero((sh == 0.0).all(axis=1))[0])
    ref = oracle_mod.phi(p, atoms, kv, kc, sh, zero, cutoff) @ q
    ew = gpu_ctx.ewald(cube.n_grid, cube.axis_vector, cutoff, kmax)
    try:
        kept = torch.from_numpy(np.ascontiguousarray(idx, dtype=np.int32)).cuda()
        V = gpu_ctx.potential(ew, atoms, q, kept).cpu().numpy()
        whole = gpu_ctx.potential(ew, atoms, q, npts=cube.n_points).cpu().numpy()
    finally:
        ew.close()
    assert np.abs(V - ref).max() <= 1e-6 * np.abs(ref).max()
    assert np.abs(whole[idx] - ref).max() <= 1e-6 * np.abs(ref).max()
