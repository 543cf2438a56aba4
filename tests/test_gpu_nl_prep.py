"""curl(u) for the nonlinear terms of a lone pipe, formed by blocks that share
the radial points of 32 modes: runs of eight points and what is left of them,
runs of more, one block for all, and the rows that a run reads beside it.

The terms against the separate vel_transform + vel_nonlinear, whose curl shares
no code with it, at the bars of the transform tests (1e-12; mixed 4e-6 of the
field's norm); and a step that imposes the mean mode's symmetry on the way
against one after vel_imposesym, bit for bit.
"""
import numpy as np
import pytest

from _util import device_pipe

pytestmark = pytest.mark.gpu

# modes / 32 chunks: 1, 3, 24 (12 runs), 127 (2 runs), 189 (one block for all)
DIMS = [(10, 4, 4), (16, 4, 4), (17, 8, 6), (33, 8, 6), (128, 4, 4), (40, 24, 16), (121, 24, 16), (65, 64, 32),
        (20, 64, 48)]


def _state(p, rng, mean_sym):
    st = []
    for _ in range(3):
        re, im = 1e-3 * rng.standard_normal((2, p.N, p.H))
        if mean_sym:
            im[:, 0] = 0.0
        st.append((re, im))
    if mean_sym:
        st[0][0][:, 0] = 0.0
    return st


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "N%dK%dM%d" % d)
def test_terms_and_mean_symmetry(dims, mixed):
    import pipeflow as P
    N, K, M = dims
    cfgd = dict(N=N, K=K, M=M, Mp=1, Re=2200.0, alpha=1.1, dt=1e-4)
    extra = {"precision": P.PF_PREC_MIXED} if mixed else {}
    a, b = device_pipe(cfgd, **extra), device_pipe(cfgd, **extra)
    rng = np.random.default_rng(17)
    a.set_state(*_state(a, rng, True))
    a.vel_transform()
    a.vel_nonlinear()
    want = [a.vel_field(3 + i).download() for i in range(3)]
    a.vel_transform_nonlinear()
    for i, (br, bi) in enumerate(want):
        ar, ai = a.vel_field(3 + i).download()
        d = np.sqrt(np.sum((ar - br) ** 2 + (ai - bi) ** 2))
        assert d <= (4e-6 if mixed else 1e-12) * np.sqrt(np.sum(br ** 2 + bi ** 2))
    st = _state(a, rng, False)
    for p in (a, b):
        p.vel_matrices()
        p.set_state(*st)
    b.vel_imposesym()
    for p in (a, b):
        p.steporbit(1)
    for (ar, ai), (br, bi) in zip(a.get_state(), b.get_state()):
        assert np.array_equal(ar, br) and np.array_equal(ai, bi)
    a.close()
    b.close()
