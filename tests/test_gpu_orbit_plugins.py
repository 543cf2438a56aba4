"""Orbit steps of a pipe that has a util plug-in or a host callback set.

Orbit steps do not call the hook (newton.f90:740-762 has none), so such a pipe
must step bit for bit like one without a plug-in, and its terms must be those
of the velocity that the predictor has just made.

Tolerance of the comparison with the separate calls: FP64 is bit for bit (both
form curl(u) alike).  In mixed precision the mean mode's sums over H modes are
taken in another order, which moves them by at most H eps of the sum of their
magnitudes, and nothing of that reaches an FP32 rounding within one step: H eps
of the state, 2.2e-16 H.
"""
import numpy as np
import pytest

from _util import device_pipe

pytestmark = pytest.mark.gpu

CFGS = [dict(N=20, K=6, M=5, Mp=1, Re=2200.0, alpha=1.1, dt=0.01),
        dict(N=40, K=24, M=16, Mp=1, Re=2000.0, alpha=1.25, dt=0.01)]
PLUGINS = ["coriolis", "carreau", "les", "callback"]


def _set(g, plugin):
    import pipeflow as P
    if plugin == "coriolis":
        g.util_set(P._lib.PF_UTIL_CORIOLIS, (0.5, 0.3))
    elif plugin == "carreau":
        g.util_set(P._lib.PF_UTIL_CARREAU_YASUDA, (1000.0, 0.01, 0.05, 0.0035, 3.3, 0.36, 2.0))
    elif plugin == "les":
        g.util_set(P._lib.PF_UTIL_LES, (1, 0.1, 1, 26.0))
    elif plugin == "callback":
        g.util_set_callback(lambda flag: None)


def _prec(mixed):
    import pipeflow as P
    return {"precision": P.PF_PREC_MIXED} if mixed else {}


def _equal(a, b):
    return all(np.array_equal(ar, br) and np.array_equal(ai, bi)
               for (ar, ai), (br, bi) in zip(a.get_state(), b.get_state()))


@pytest.mark.parametrize("cfgd", CFGS, ids=["small", "cfg1"])
@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("plugin", PLUGINS)
def test_orbit_steps_do_not_feel_a_plugin(cfgd, mixed, plugin):
    import pipeflow as P
    a, b, c = (device_pipe(cfgd, **_prec(mixed)) for _ in range(3))
    _set(a, plugin)
    for p in (a, b, c):
        p.vel_matrices()
    P.seeded_state(b, 9, 1e-3)
    for p in (a, c):
        p.set_state(*b.get_state())
    a.steporbit(1)
    b.steporbit(1)
    assert _equal(a, b)
    c.vel_imposesym()
    c.vel_transform_nonlinear()
    c.vel_predictor()
    c.vel_transform_nonlinear()
    c.vel_corrector()
    c.vel_imposesym()
    x, y = (np.concatenate([np.ravel(v) for f in p.get_state() for v in f]) for p in (a, c))
    tol = 2.2e-16 * a.H if mixed else 0.0
    assert np.linalg.norm(x - y) <= tol * np.linalg.norm(y)
    a.steporbit(2)
    b.steporbit(2)
    assert _equal(a, b)
    for p in (a, b, c):
        p.close()


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
def test_an_orbit_batch_with_a_plugin_equals_one_without(mixed):
    import pipeflow as P
    cfgs = [P.PipeConfig(**d, **_prec(mixed)) for d in (CFGS[0], CFGS[1], CFGS[0])]
    a, b = P.Batch(cfgs), P.Batch(cfgs)
    for batch in (a, b):
        batch.matrices()
        for i, p in enumerate(batch.pipes):
            P.seeded_state(p, 30 + i, 1e-3)
    a.step(1, orbit=True)  # launches built before the plug-in is set
    b.step(1, orbit=True)
    _set(a.pipes[1], "coriolis")
    for _ in range(2):
        a.step(1, orbit=True)
        b.step(1, orbit=True)
    for pa, pb in zip(a.pipes, b.pipes):
        assert _equal(pa, pb)
    a.close()
    b.close()
