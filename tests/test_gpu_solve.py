"""The bordered solve at the sizes where its blocking can go wrong: one unknown, the 32-column panel's
edges, the change of thread counts at 100 unknowns, the last size one CTA factors; on matrices that need row
interchanges in every panel.  Against an FP64 LU of the same bordered system, within the
bound of the other solve tests (1e-9 of the largest charge)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(A, b, qtot):
    import scipy.linalg as sl
    N = len(b)
    K = np.zeros((N + 1, N + 1))
    K[:N, :N] = A
    K[:N, N] = K[N, :N] = 1.0
    return K, sl.solve(K, np.append(b, qtot))[:N]


@pytest.mark.parametrize("N", [1, 2, 30, 31, 32, 33, 62, 63, 64, 65, 99, 100, 255, 256, 513, 766])
def test_pivoted_systems_at_panel_edges(N, gpu_ctx):
    """Symmetric indefinite A with a weak diagonal: the pivot is off the diagonal in most columns."""
    import torch
    rng = np.random.default_rng(N)
    A = rng.normal(size=(N, N))
    A = 0.5 * (A + A.T)
    A[np.arange(N), np.arange(N)] *= 0.01
    A += np.diag(np.where(np.arange(N) % 7 == 0, 3.0, 0.0))
    b = rng.normal(size=N)
    K, ref = _reference(A, b, 0.25)
    q, info = gpu_ctx.solve(torch.from_numpy(A).cuda(), torch.from_numpy(b).cuda(), np.full(N, 6), qtot=0.25)
    q = q.cpu().numpy()
    tol = max(1e-9, 1e-15 * np.linalg.cond(K) * (N + 1))
    assert np.abs(q - ref).max() <= tol * max(1.0, np.abs(ref).max())
    kappa = np.abs(A).sum(axis=0).max() * np.abs(np.linalg.inv(K)).sum(axis=0).max()
    assert kappa / 3 <= info["kappa"] <= kappa * (1 + 1e-3)


@pytest.mark.parametrize("N", [5, 40])
def test_nan_matrix_is_reported_singular_or_nan(N, gpu_ctx):
    """A matrix of NaN has no pivot: the solve ends, and returns no finite charge as if it were one."""
    import torch
    from pyrepeat_gb300 import _lib
    A = torch.full((N, N), float("nan"), dtype=torch.float64, device="cuda")
    b = torch.zeros(N, dtype=torch.float64, device="cuda")
    try:
        q, _ = gpu_ctx.solve(A, b, np.full(N, 6))
    except _lib.RepeatError:
        return
    assert not np.isfinite(q.cpu().numpy()).all()


@pytest.mark.parametrize("N", [767, 800, 1023, 1055, 2047, 2049, 2600, 4095, 4096])
def test_wide_pivoted_systems(N, gpu_ctx):
    """The factorisation across the GPU: the changes of its panel width at 1024 and 2048 rows, its last
    size and the first beyond it.  The bound of the test above, with the 1-norm condition number."""
    import torch
    rng = np.random.default_rng(N)
    A = rng.normal(size=(N, N))
    A = 0.5 * (A + A.T)
    A[np.arange(N), np.arange(N)] *= 0.01
    b = rng.normal(size=N)
    K, ref = _reference(A, b, 0.25)
    q, _ = gpu_ctx.solve(torch.from_numpy(A).cuda(), torch.from_numpy(b).cuda(), np.full(N, 6), qtot=0.25)
    q = q.cpu().numpy()
    kinv = np.abs(np.linalg.inv(K)).sum(axis=0).max()
    tol = max(1e-9, 1e-15 * np.abs(K).sum(axis=0).max() * kinv * (N + 1))
    assert np.abs(q - ref).max() <= tol * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("N", [300, 800])
def test_singular_systems_across_the_gpu(N, gpu_ctx):
    """Two equal rows and columns: refused as singular, or solved with a residual that says so."""
    import torch
    from pyrepeat_gb300 import _lib
    rng = np.random.default_rng(N)
    A = rng.normal(size=(N, N))
    A = A @ A.T / N
    A[:, N // 2] = A[:, 3]
    A[N // 2, :] = A[3, :]
    try:
        _, info = gpu_ctx.solve(torch.from_numpy(A).cuda(), torch.from_numpy(rng.normal(size=N)).cuda(), np.full(N, 6))
    except _lib.RepeatError:
        return
    assert info["kappa"] > 1e12


@pytest.mark.parametrize("where", [5, 2000, 4190])
def test_zero_pivot_in_the_panels_beyond_the_register_panels(where, gpu_ctx):
    """Two atoms without any normal-equation entries leave an exactly zero pivot, here in the first, a middle
    and the last panel of a system factored by panels in shared memory, whose later panels then write no
    interchanges: reported singular, and the context solves the next system."""
    import torch
    from pyrepeat_gb300 import _lib
    N = 4200
    g = torch.Generator(device="cuda").manual_seed(where)
    A = torch.randn(N, N, generator=g, dtype=torch.float64, device="cuda") / N
    A = A + A.T + 10.0 * torch.eye(N, dtype=torch.float64, device="cuda")  # (the border is no pivot but theirs)
    good = A.clone()
    for i in (where, where + 3):
        A[i, :] = 0.0
        A[:, i] = 0.0
    b = torch.randn(N, generator=g, dtype=torch.float64, device="cuda")
    with pytest.raises(_lib.RepeatError):
        gpu_ctx.solve(A, b, np.full(N, 6))
    q, _ = gpu_ctx.solve(good, b, np.full(N, 6))
    K = torch.ones(N + 1, N + 1, dtype=torch.float64, device="cuda")
    K[:N, :N] = good
    K[N, N] = 0.0
    ref = torch.linalg.solve(K, torch.cat([b, b.new_zeros(1)]))[:N]
    assert float((q - ref).abs().max()) <= 1e-10 * float(ref.abs().max())


@pytest.mark.parametrize("N", [255, 382, 383, 384, 511, 766, 1151, 1152])
def test_refinement_across_the_gpu(N, gpu_ctx):
    """One system refined across the GPU, at the edges of its 128-unknown blocks, for a matrix whose
    solution and condition estimate are checked against FP64.  The estimate is Hager's with FP32
    solves, whose relative error is below n eps32 kappa."""
    import torch
    rng = np.random.default_rng(N)
    X = rng.normal(size=(3 * N, N))
    A = X.T @ X / (3 * N)
    b = rng.normal(size=N)
    K, ref = _reference(A, b, -1.5)
    q, info = gpu_ctx.solve(torch.from_numpy(A).cuda(), torch.from_numpy(b).cuda(), np.full(N, 6), qtot=-1.5)
    q = q.cpu().numpy()
    kinv = np.abs(np.linalg.inv(K)).sum(axis=0).max()
    kk = np.abs(K).sum(axis=0).max() * kinv
    assert np.abs(q - ref).max() <= max(1e-12, 1e-15 * kk * (N + 1)) * max(1.0, np.abs(ref).max())
    kappa = np.abs(A).sum(axis=0).max() * kinv
    assert kappa / 3 <= info["kappa"] <= kappa * (1 + (N + 1) * 2.0**-24 * kk)
    xmax = np.abs(np.linalg.solve(K, np.append(b, -1.5))).max()
    assert info["residual"] <= 2 * (N + 1) * 2.0**-53 * np.abs(K).sum(axis=0).max() * xmax


@pytest.mark.parametrize("N", [769, 830, 895, 1025, 1100, 1151, 1281])
def test_repeated_solves_agree_on_a_busy_gpu(N, gpu_ctx):
    """Odd numbers of 128-unknown blocks, whose two sweeps meet in one exchange buffer: charges and kappa of
    repeated solves are the same bits while another stream keeps the SMs busy."""
    import torch
    rng = np.random.default_rng(N)
    X = rng.normal(size=(2 * N, N))
    A = torch.from_numpy(X.T @ X / (2 * N)).cuda()
    b = torch.from_numpy(rng.normal(size=N)).cuda()
    side = torch.cuda.Stream()
    a = torch.rand(1 << 22, device="cuda")
    m = torch.rand(1536, 1536, device="cuda")
    seen = []
    for rep in range(12):
        with torch.cuda.stream(side):
            for _ in range(4 * (rep % 4)):
                a = a * 0.999 + 0.001
                m = (m @ m).clamp_(0.0, 1.0)
        q, info = gpu_ctx.solve(A, b, np.full(N, 6), qtot=0.5)
        seen.append((q.cpu().numpy().tobytes(), info["kappa"]))
    torch.cuda.synchronize()
    assert len(set(seen)) == 1


@pytest.mark.parametrize("N", [400, 900])
def test_slow_refinement(N, gpu_ctx):
    """kappa towards 1/eps32: refinement with inverted blocks, by substitution, and FP64 factors."""
    import torch
    rng = np.random.default_rng(7)
    U, _ = np.linalg.qr(rng.normal(size=(N, N)))
    for top in (1e5, 1e6, 1e7, 1e9):
        A = (U * np.geomspace(1.0 / top, 1.0, N)) @ U.T
        A = 0.5 * (A + A.T)
        b = rng.normal(size=N)
        K, ref = _reference(A, b, 0.0)
        q, info = gpu_ctx.solve(torch.from_numpy(A).cuda(), torch.from_numpy(b).cuda(), np.full(N, 6), qtot=0.0)
        tol = max(1e-12, 1e-15 * np.linalg.cond(K) * (N + 1))
        assert np.abs(q.cpu().numpy() - ref).max() <= tol * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("N", [400, 900])
def test_solve_within_a_tight_scratch_budget(N):
    """Room for the system and its copy, not for the factors' extra buffer: solved by the ways that need none."""
    import torch
    from pyrepeat_gb300.fit import Context
    rng = np.random.default_rng(N)
    X = rng.normal(size=(3 * N, N))
    A = X.T @ X / (3 * N)
    b = rng.normal(size=N)
    K, ref = _reference(A, b, 0.5)
    ctx = Context(0, hbm_budget=16 * (N + 1) ** 2 + (2 << 20))
    q, _ = ctx.solve(torch.from_numpy(A).cuda(), torch.from_numpy(b).cuda(), np.full(N, 6), qtot=0.5)
    tol = max(1e-12, 1e-15 * np.linalg.cond(K) * (N + 1))
    assert np.abs(q.cpu().numpy() - ref).max() <= tol * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("N", [420, 900, 2040])
def test_charges_do_not_depend_on_the_scratch_left(N, gpu_ctx):
    """The same system in a context with room for it alone and in one with all of the memory: the same bits."""
    import torch
    from pyrepeat_gb300.fit import Context
    rng = np.random.default_rng(N)
    A = rng.normal(size=(N, N))
    A = 0.5 * (A + A.T) + np.diag(np.where(np.arange(N) % 5 == 0, 40.0, 0.0))
    A, b = torch.from_numpy(A).cuda(), torch.from_numpy(rng.normal(size=N)).cuda()
    tight = Context(0, hbm_budget=16 * (N + 1) ** 2 + (2 << 20))
    out = [(q.cpu().numpy().tobytes(), info["kappa"])
           for q, info in (c.solve(A, b, np.full(N, 6), qtot=0.25) for c in (tight, gpu_ctx))]
    assert out[0] == out[1]


@pytest.mark.parametrize("N", [3, 40, 200])
@pytest.mark.parametrize("top", [1e2, 1e10])
def test_systems_with_their_vectors_in_memory(N, top, gpu_ctx):
    """What systems beyond 11520 unknowns run (their vectors do not fit shared memory), at sizes that take no
    minutes: by FP32 factors and refinement, and by FP64 factors.  The bound of the first test."""
    import ctypes
    import torch
    hook = gpu_ctx.lib.rp_debug_solve_in_memory
    hook.restype, hook.argtypes = ctypes.c_int, [ctypes.c_void_p, ctypes.c_int]
    rng = np.random.default_rng(N)
    U, _ = np.linalg.qr(rng.normal(size=(N, N)))
    A = (U * np.geomspace(1.0 / top, 1.0, N)) @ U.T
    A = 0.5 * (A + A.T)
    b = rng.normal(size=N)
    K, ref = _reference(A, b, 0.25)
    assert hook(gpu_ctx.ptr, 1) == 0
    try:
        q, info = gpu_ctx.solve(torch.from_numpy(A).cuda(), torch.from_numpy(b).cuda(), np.full(N, 6), qtot=0.25)
    finally:
        hook(gpu_ctx.ptr, 0)
    tol = max(1e-9, 1e-15 * np.linalg.cond(K) * (N + 1))
    assert np.abs(q.cpu().numpy() - ref).max() <= tol * max(1.0, np.abs(ref).max())
