"""Charges do not depend on the batch: cubes whose systems (256 to 767 unknowns) may be factored in one CTA
or across the GPU, fitted alone, in pairs, in larger batches and served, give the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RESP = {s: (0.1, 0.0) for s in ("H", "C", "N", "O", "S", "Zn")}


def _cube(n, ctx):
    from pyrepeat_gb300 import synth
    cube = synth.make_tric(seed=n, n_grid=(60, 56, 63), n_atoms=n, n_groups=0, ctx=ctx)
    cube.resp = RESP
    return cube


@pytest.mark.parametrize("n", [256, 300, 430, 590, 700])
def test_mid_size_systems_alone_and_in_batches(n, gpu_ctx):
    from pyrepeat_gb300 import _lib
    cubes = {m: _cube(m, gpu_ctx) for m in (n, n + 20, n + 35, 60)}

    def fit(names, submit=False):
        cs = [cubes[m] for m in names]
        V = [c.V_dev for c in cs]
        if submit:
            q, _, info = gpu_ctx.batch_submit(cs, _lib.PREC_MIXED, V_dev=V).result()
        else:
            q, _, info = gpu_ctx.fit_batch(cs, _lib.PREC_MIXED, V_dev=V)
        return [(np.array(a).tobytes(), _lib.fit_info(i)["kappa"]) for a, i in zip(q, info)]

    alone = {m: fit([m])[0] for m in cubes}
    for names in ([n, n + 20], [60, n], [n, n + 20, n + 35], [n + 35] * 7 + [n, 60]):
        for submit in (False, True):
            for m, got in zip(names, fit(names, submit)):
                assert got == alone[m], (m, names, submit)


@pytest.mark.parametrize("vdw", [1.0, 1.2, 1.3])
def test_ill_conditioned_systems_alone_and_in_batches(vdw, gpu_ctx):
    """Systems that need more rounds, substitution or FP64 factors (no escalation), in a launch with more of them
    than one set of the rounds holds."""
    from pyrepeat_gb300 import _lib
    cubes = [_cube(n, gpu_ctx) for n in (270, 411, 440, 520)]
    for c, t in zip(cubes, (0.1, 1e-3, 1e-5, 0.0)):
        c.vdw_factor = vdw
        c.resp = {s: (t, 0.0) for s in RESP} if t else None
    gpu_ctx.set_kappa_limit(0.0)
    try:
        alone = []
        for c in cubes:
            q, _, info = gpu_ctx.fit_batch([c], _lib.PREC_MIXED, V_dev=[c.V_dev])
            alone.append((np.array(q[0]).tobytes(), _lib.fit_info(info[0])["kappa"]))
        which = [0, 1, 2, 3] * 5 + [2]
        q, _, info = gpu_ctx.fit_batch([cubes[k] for k in which], _lib.PREC_MIXED, V_dev=[cubes[k].V_dev for k in which])
    finally:
        gpu_ctx.set_kappa_limit(_lib.DEFAULT_KAPPA_LIMIT)
    for k, a, i in zip(which, q, info):
        assert (np.array(a).tobytes(), _lib.fit_info(i)["kappa"]) == alone[k], k
    print([_lib.fit_info(i)["solve_path"] for i in info[:4]], ["%.1e" % _lib.fit_info(i)["kappa"] for i in info[:4]])
