"""The Phi kernel at the edges of its tiles: 128 points per CTA in pairs, atoms in blocks, E values
staged per run of points in one grid row (four atoms at a time up to 32 runs, two up to
64, one beyond), an image table that a tile may overflow.  Against the oracle's FP64 Phi of the
same points, within the 1e-6 of max|Phi| that every mixed Phi value is held to."""
import ctypes

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


def _phi(ctx, cube, atoms, idx, kmax, parts=3):
    import torch
    L = ctx.lib
    L.rp_debug_mixed_phi.restype = ctypes.c_int
    L.rp_debug_mixed_phi.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int,
                                     ctypes.c_void_p, ctypes.c_int64, ctypes.c_int, ctypes.c_void_p]
    ew = ctx.ewald(cube.n_grid, cube.axis_vector, cube.cutoff, kmax)
    kept = torch.from_numpy(np.ascontiguousarray(idx, dtype=np.int32)).cuda()
    out = torch.zeros((len(atoms), len(idx)), dtype=torch.float64, device="cuda")
    try:
        ctx.check(L.rp_debug_mixed_phi(ctx.ptr, ew.ptr, atoms.ctypes.data, len(atoms), kept.data_ptr(), len(idx),
                                       parts, out.data_ptr()))
    finally:
        ew.close()
    return out.cpu().numpy().T


def _reference(oracle_mod, cube, atoms, idx, kmax):
    from pyrepeat_gb300 import synth
    nx, ny = int(cube.n_grid[0]), int(cube.n_grid[1])
    i, j, k = idx % nx, (idx // nx) % ny, idx // (nx * ny)
    g = i[:, None] * cube.axis_vector[0] + j[:, None] * cube.axis_vector[1] + k[:, None] * cube.axis_vector[2]
    box = cube.box_vectors
    _, kv, kc = synth.kspace(box, cube.cutoff, kmax)
    sh = synth.realspace_shifts(box, cube.cutoff)
    zero = int(np.flatnonzero((sh == 0.0).all(axis=1))[0])
    return oracle_mod.phi(g, atoms, kv, kc, sh, zero, cube.cutoff)


def _check(got, ref):
    assert np.abs(got - ref).max() <= 1e-6 * np.abs(ref).max()


@pytest.mark.parametrize("kmax", [7, 3])
@pytest.mark.parametrize("n,rows,order", [(1, 1, "flat"), (1, 127, "flat"), (2, 128, "shuffled"), (9, 129, "flat"),
                                          (31, 66, "shuffled"), (33, 257, "flat"), (40, 384, "shuffled"),
                                          (37, 250, "pairs")])
def test_phi_at_tile_edges(n, rows, order, kmax, gpu_ctx, oracle_mod):
    cube, g = load_golden("tricmini")
    atoms = np.ascontiguousarray(cube.atom_pos[:n], dtype=np.float64)
    idx = np.flatnonzero(g["mask"])
    if order != "flat":
        idx = np.random.default_rng(n).permutation(idx)
    if order == "pairs":  # runs of two points: more than 32 and at most 64 or so per tile
        idx = np.stack([idx[:rows], np.minimum(idx[:rows] + 1, cube.n_points - 1)], axis=1).ravel()
    idx = idx[:rows]
    _check(_phi(gpu_ctx, cube, atoms, idx, kmax), _reference(oracle_mod, cube, atoms, idx, kmax))


@pytest.mark.parametrize("n", [7, 32])
def test_phi_small_cell_overflows_the_image_table(n, gpu_ctx, oracle_mod):
    """A 12 Bohr cell: ~9 of its up to 125 images per atom are within the cutoff of a point, and
    a tile of points spread over the cell reaches several times as many."""
    from pyrepeat_gb300 import synth
    rng = np.random.default_rng(3)
    ng = np.array([40, 41, 43])
    cell = np.diag([12.0, 12.5, 13.0])
    atoms = np.ascontiguousarray(rng.random((n, 3)) @ cell)
    cube = synth.Cube(np.full(n, 6), atoms, ng, cell / ng[:, None], None)
    idx = rng.permutation(cube.n_points)[:300]
    nx, ny = int(ng[0]), int(ng[1])
    p = np.stack([idx % nx, (idx // nx) % ny, idx // (nx * ny)], axis=1) @ cube.axis_vector
    far = np.ones(len(idx), bool)  # points at least 1 Bohr from every image, as after a vdW filter
    for s in synth.realspace_shifts(cell, 1.0):
        far &= (np.linalg.norm(p[:, None] - (atoms + s)[None], axis=2) > 1.0).all(axis=1)
    idx = idx[far]
    _check(_phi(gpu_ctx, cube, atoms, idx, 7), _reference(oracle_mod, cube, atoms, idx, 7))


@pytest.mark.parametrize("kmax", [1, 2, 6, 12, 20])
@pytest.mark.parametrize("n", [1, 17, 34])
def test_phi_over_kmax(n, kmax, gpu_ctx, oracle_mod):
    """The reciprocal rows' stages: columns of more entries than one CTA's slab, an odd and an even number
    of columns, one n1, rows that are no multiple of eight."""
    cube, g = load_golden("tricmini")
    atoms = np.ascontiguousarray(cube.atom_pos[:n], dtype=np.float64)
    idx = np.random.default_rng(kmax).permutation(cube.n_points)[:300].astype(np.int64)
    idx = idx[g["mask"].ravel()[idx] != 0]
    _check(_phi(gpu_ctx, cube, atoms, idx, kmax), _reference(oracle_mod, cube, atoms, idx, kmax))


@pytest.mark.parametrize("n_grid,n_atoms", [((80, 85, 90), 300), ((96, 75, 64), 200), ((110, 121, 63), 420)])
def test_fits_of_crowded_cells(n_grid, n_atoms, gpu_ctx):
    """A batch writes only the grid rows near kept points in a crowded cell.  The mixed fit against the
    FP64 fit of the same cube, after a fit of another cube has left its rows in the scratch, within
    ten times the usual distance of the two (2e-11 kappa / (n + 1) e)."""
    from pyrepeat_gb300 import _lib, synth
    s = (n_atoms / 2000.0) ** (1 / 3)
    cubes = [synth.make_tric(seed=k, n_grid=n_grid, n_atoms=n_atoms, n_groups=10,
                             lengths=(40.0 * s, 42.0 * s, 45.0 * s), ctx=gpu_ctx) for k in (5, 6)]
    gpu_ctx.set_kappa_limit(0.0)
    try:
        q = []
        for c, prec in ((cubes[1], _lib.PREC_MIXED), (cubes[0], _lib.PREC_MIXED), (cubes[0], _lib.PREC_FP64)):
            r, _, info = gpu_ctx.fit_batch([c], prec, V_dev=[c.V_dev] if c.V is None else None)
            q.append(np.asarray(r[0]).copy())
    finally:
        gpu_ctx.set_kappa_limit(_lib.DEFAULT_KAPPA_LIMIT)
    kappa = _lib.fit_info(info[0])["kappa"]
    assert np.abs(q[1] - q[2]).max() <= max(1e-5, 2e-10 * kappa / (n_atoms + 1)) * max(1.0, np.abs(q[2]).max())
