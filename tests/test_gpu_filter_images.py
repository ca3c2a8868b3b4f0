"""The filter's choice of lattice images: only those that can reject a point are carried where every point
is proved near, all effective ones otherwise.  Against the rule itself, image by image in FP64:
cells of any shape, atoms inside and outside them, factors from nothing to beyond the cell."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rule(n_grid, axis, atoms, radius, factor, vmax):
    box = axis * n_grid[:, None]
    corners = np.array([(i * axis[0] + j * axis[1]) + k * axis[2] for i in (0, 1) for j in (0, 1) for k in (0, 1)])
    margin = vmax * radius.max() + 0.1
    i, j, k = np.meshgrid(*(np.arange(n) for n in n_grid), indexing="ij")
    g = (i[..., None] * axis[0] + j[..., None] * axis[1]) + k[..., None] * axis[2]
    keep, near = np.ones(i.shape, bool), np.zeros(i.shape, bool)
    for a, r in zip(atoms, radius):
        for kz in (-1, 0, 1):
            for ky in (-1, 0, 1):
                for kx in (-1, 0, 1):
                    e = a + ((kx * box[0] + ky * box[1]) + kz * box[2])
                    if not ((e >= corners.min(0) - margin).all() and (e <= corners.max(0) + margin).all()):
                        continue
                    d = g - e
                    d2 = (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2]
                    keep &= d2 > (factor * r) ** 2
                    near |= d2 <= (vmax * r) ** 2
    return np.flatnonzero((keep & near).transpose(2, 1, 0).ravel())  # flat index: first axis fastest


@pytest.mark.parametrize("factor,vmax", [(1.0, 1000.0), (0.0, 1000.0), (0.4, 1000.0), (4.0, 1000.0), (0.7, 2.0), (0.7, 0.8)])
@pytest.mark.parametrize("cell", ["cubic", "slanted", "flat", "far"])
def test_kept_points_follow_the_rule(cell, factor, vmax, gpu_ctx):
    import torch
    rng = np.random.default_rng(len(cell))
    axis = {"cubic": np.diag([0.5, 0.5, 0.5]), "slanted": np.array([[0.5, 0, 0], [-0.3, 0.45, 0], [0.2, -0.25, 0.5]]),
            "flat": np.diag([0.9, 0.02, 0.7]), "far": np.diag([0.4, 0.5, 0.6])}[cell]
    n_grid = np.array([23, 18, 27])
    box = axis * n_grid[:, None]
    atoms = rng.random((5, 3)) @ box
    if cell == "far":
        atoms += np.array([2.6, 0.0, -1.4]) @ box  # whole cells away: images at one cell reach some points only
    Z = np.array([1, 6, 8, 30, 16])
    radius = np.array([2.72687, 3.63867, 3.30702, 2.61066, 3.81252])  # Bohr, the filter's table
    V = torch.from_numpy(rng.normal(size=int(np.prod(n_grid)))).cuda()
    ref = _rule(n_grid, axis, atoms, radius, factor, vmax)
    if len(ref) == 0:
        pytest.skip("no point is kept")
    kept, _, M, _ = gpu_ctx.filter(n_grid, axis, atoms, Z, V, factor, vmax)
    got = np.sort(kept.cpu().numpy()[:int(M)])
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("cell", ["cubic", "slanted", "flat", "far"])
def test_no_point_is_kept_where_the_rule_keeps_none(cell, gpu_ctx):
    """The same cells at factors up to spheres that cover them: where the rule rejects every point, so does the
    filter."""
    import torch
    axis = {"cubic": np.diag([0.5, 0.5, 0.5]), "slanted": np.array([[0.5, 0, 0], [-0.3, 0.45, 0], [0.2, -0.25, 0.5]]),
            "flat": np.diag([0.9, 0.02, 0.7]), "far": np.diag([0.4, 0.5, 0.6])}[cell]
    n_grid = np.array([23, 18, 27])
    box = axis * n_grid[:, None]
    rng = np.random.default_rng(len(cell))
    atoms = rng.random((5, 3)) @ box
    if cell == "far":
        atoms += np.array([2.6, 0.0, -1.4]) @ box
    Z = np.array([1, 6, 8, 30, 16])
    radius = np.array([2.72687, 3.63867, 3.30702, 2.61066, 3.81252])
    V = torch.from_numpy(rng.normal(size=int(np.prod(n_grid)))).cuda()
    empty = 0
    for factor, vmax in ((4.0, 1000.0), (8.0, 1000.0), (1.0, 0.9), (4.0, 3.0)):
        if len(_rule(n_grid, axis, atoms, radius, factor, vmax)) == 0:
            empty += 1
            assert gpu_ctx.filter(n_grid, axis, atoms, Z, V, factor, vmax)[2] == 0, (factor, vmax)
    assert empty > 0
