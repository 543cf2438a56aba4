"""The transform launches of the nonlinear terms at every built length, in
both precisions, against the separate vel_transform + vel_nonlinear (generic
FP64 kernels that share no code with them), and the curl a fused predictor
leaves against the one formed from its velocity.

Tolerances: FP64, the bar of the transform tests, 1e-12.  Mixed precision: a
coefficient passes three FP32 transforms of at most log2(384) < 9 levels, a
product and two roundings into FP32, each level growing the error by about one
unit in the last place of the row's norm: 30 * 2^-24 < 2e-6, doubled for the
spread between the three components; 4e-6 of the field's norm.
"""
import numpy as np
import pytest

from _util import device_pipe

pytestmark = pytest.mark.gpu

# every built 3K and 3M, with odd and even column counts in a z-pass tile
PAIRS = [(4, 128), (5, 96), (6, 64), (8, 48), (12, 32), (16, 24), (24, 16), (32, 12), (48, 8), (64, 6), (96, 5),
         (128, 4), (128, 48), (64, 32)]


def _N(pipe):
    return [pipe.vel_field(3 + i).download() for i in range(3)]


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("km", PAIRS, ids=lambda p: "K%dM%d" % p)
def test_nonlinear_terms_at_every_length(km, mixed):
    import pipeflow as P
    K, M = km
    cfgd = dict(N=11, K=K, M=M, Mp=1, Re=2200.0, alpha=1.1, dt=0.01)
    g = device_pipe(cfgd, **({"precision": P.PF_PREC_MIXED} if mixed else {}))
    rng = np.random.default_rng(7)
    st = []
    for _ in range(3):  # every mode alive, the mean one real
        re, im = rng.standard_normal((2, g.N, g.H))
        im[:, 0] = 0.0
        st.append((re, im))
    st[0][0][:, 0] = 0.0
    g.set_state(*st)
    g.vel_transform()
    g.vel_nonlinear()
    want = _N(g)
    g.vel_transform_nonlinear()
    got = _N(g)
    tol = 4e-6 if mixed else 1e-12
    for (ar, ai), (br, bi) in zip(got, want):
        d = np.sqrt(np.sum((ar - br) ** 2 + (ai - bi) ** 2))
        assert d <= tol * np.sqrt(np.sum(br ** 2 + bi ** 2))
    g.close()


@pytest.mark.parametrize("dims", [dict(N=17, K=6, M=5, Mp=2), dict(N=40, K=24, M=16), dict(N=65, K=4, M=4)],
                         ids=lambda d: "N{N}K{K}M{M}".format(**d))
def test_curl_left_by_the_predictor_equals_the_curl_of_its_velocity(dims):
    import pipeflow as P
    cfgd = {**dict(Mp=1, Re=2200.0, alpha=1.1, dt=0.01), **dims}
    a, b = device_pipe(cfgd), device_pipe(cfgd)
    for p in (a, b):
        p.vel_matrices()
    P.seeded_state(a, 9, 1e-3)
    b.set_state(*a.get_state())
    a.steporbit(1)  # the predictor's curl feeds the corrector's terms
    b.vel_imposesym()
    b.vel_transform_nonlinear()
    b.vel_predictor()
    b.vel_transform_nonlinear()
    b.vel_corrector()
    b.vel_imposesym()
    for (ar, ai), (br, bi) in zip(a.get_state(), b.get_state()):
        assert np.array_equal(ar, br) and np.array_equal(ai, bi)
    a.close()
    b.close()
