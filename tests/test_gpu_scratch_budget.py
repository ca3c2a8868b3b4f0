"""FP64 normal equations and QEq within a scratch budget that holds no more than a flat table of the wave
vectors would: the stages work block by block, and the results have the bits of an ample budget."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cell(n, n_grid, seed):
    rng = np.random.default_rng(seed)
    box = np.array([[18.0, 0.0, 0.0], [1.5, 19.0, 0.0], [-1.0, 2.0, 20.0]])
    return box / np.array(n_grid)[:, None], rng.random((n, 3)) @ box, rng


@pytest.mark.parametrize("n,kmax,n_grid,M", [(300, 9, (40, 44, 160), 1500), (33, 7, (30, 32, 500), 700),
                                             (200, 0, (40, 40, 40), 20000), (17, 0, (40, 40, 40), 60000),
                                             (130, 12, (64, 64, 64), 100)])
def test_fp64_gram_in_a_tight_budget(n, kmax, n_grid, M, gpu_ctx):
    import torch
    from pyrepeat_gb300 import _lib
    from pyrepeat_gb300.fit import Context
    axis, atoms, rng = _cell(n, n_grid, n)
    kept = torch.from_numpy(np.sort(rng.permutation(int(np.prod(n_grid)))[:M]).astype(np.int32)).cuda()
    V = torch.from_numpy(rng.normal(size=M)).cuda()
    ew = gpu_ctx.ewald(n_grid, axis, 20.0, kmax)
    K = ew.K
    budget = 16 * K * n + (16 * K + 8 * n) * M + 8 * n * n + (8 << 20)
    out = []
    for ctx in (gpu_ctx, Context(0, hbm_budget=budget)):
        e = ctx.ewald(n_grid, axis, 20.0, kmax)
        out.append([t.cpu().numpy() for t in ctx.gram(e, atoms, kept, V, _lib.PREC_FP64, want_sum_phi=True)])
        e.close()
    ew.close()
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)


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
