"""vel_matrices in a few launches: factor sets, unit solutions and influence
matrices where the register window and the four-column read-ahead can go wrong
(N on each side of a multiple of four, the least N, one mode, m = 0 alone,
pivoting factors), and again after a change of dt, which keeps the pressure set.

Tolerance: the repository's bars for these quantities (factors 1e-13 with equal
interchanges, U1..U3 1e-12; U4..U6 and the inverted matrices 1e-10, through the
nearly singular pressure systems), at sizes of the same range.
"""
import numpy as np
import pytest

import pipeflow_oracle as O
from _util import device_pipe, oracle_pipe, rel

pytestmark = pytest.mark.gpu

SIZES = [
    dict(N=10, K=3, M=1), dict(N=11, K=1, M=4), dict(N=12, K=5, M=3, Mp=2), dict(N=13, K=9, M=4, const_flux=False),
    dict(N=33, K=4, M=3), dict(N=64, K=4, M=4),
]


@pytest.mark.parametrize("dims", SIZES, ids=lambda d: "N{N}K{K}M{M}".format(**d))
def test_matrices(dims):
    cfgd = {**dict(Mp=1, Re=1900.0, alpha=1.25, dt=0.02), **dims}
    o, g = oracle_pipe({**cfgd, "dt": 0.01}), device_pipe(cfgd)
    g.vel_matrices()
    t = g.tim
    t.dt = 0.01
    g.set_tim(t)
    g.vel_matrices()  # the sets of the new dt, the pressure set kept
    fresh = device_pipe({**cfgd, "dt": 0.01})
    fresh.vel_matrices()
    o.vel_matrices()
    U, A = g.influence()
    for c in range(3):
        assert rel(U[c].T, o._U[c]) < 1e-12, c
    # one velocity field: at k = 0 its u+ is zero (p = r^m), rounding on either side
    assert rel(np.moveaxis(U[3:], 1, 2), np.stack(o._U[3:])) < 1e-10
    assert rel(A[1:], o._A[1:]) < 1e-10
    for a, b in zip((U, A), fresh.influence()):
        assert np.array_equal(a, b)
    c1, c2 = 1.0 / 0.01, -g.cfg.implicit / g.cfg.Re
    for PM, BC, a, b in ((0, 1, 0.0, 1.0), (1, 0, c1, c2), (-1, 0, c1, c2), (0, 0, c1, c2)):
        M, piv = g.tim_lumesh_init(PM, BC, a, b).download()
        ref, ref_piv = o.tim_lumesh_init(PM, BC, a, b)
        for nh in range(1 if BC else 0, o.H):
            assert np.array_equal(piv[nh] - 1, ref_piv[nh]), (PM, BC, nh)
            assert rel(M[nh].T, ref[nh]) < 1e-13
    st = O.seeded_state(o, 5, 1e-3)
    ends = []
    for p in (g, fresh):  # the tiles and the mean-flux response, through a step
        p.set_state(*[(c.re, c.im) for c in st])
        p.steporbit(2)
        ends.append(p.get_state())
    for a, b in zip(*ends):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
