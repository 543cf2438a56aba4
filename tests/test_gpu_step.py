"""The fused vel_step (one launch per predictor or corrector) at the edges of
its tiles: radial sizes on both sides of each launch shape, mode counts that
leave tiles of 8 and 16 part-filled, a pipe of m = 0 modes alone, grids smaller
and larger than the GPU, pivoting Helmholtz factors.  One predictor and two
corrector passes against the oracle, and the lone launch against the batched
one bit for bit.

Tolerance: both sides solve the same banded systems in FP64 with different
orders of rounding, so they differ by a multiple of eps times the condition of
the radial Laplacian, which grows as the fourth power of N (the wall spacing of
the mesh goes as 1/N^2); the repository's bar of 1e-12 at N <= 64 therefore
becomes 1e-12 (N/64)^4 beyond it.
"""
import numpy as np
import pytest

import pipeflow_oracle as O
from _util import device_pipe, oracle_pipe, state_from_dev, state_to_dev

pytestmark = pytest.mark.gpu

SIZES = [
    dict(N=10, K=4, M=1), dict(N=11, K=1, M=4), dict(N=16, K=18, M=2), dict(N=31, K=5, M=3),
    dict(N=32, K=16, M=4), dict(N=33, K=9, M=5, Mp=3), dict(N=47, K=3, M=6), dict(N=64, K=8, M=4),
    dict(N=65, K=7, M=3), dict(N=97, K=4, M=3), dict(N=128, K=4, M=4),
]


def _cfg(d):
    return {**dict(Mp=1, Re=2200.0, alpha=1.1, dt=0.01), **d}


@pytest.mark.parametrize("dims", SIZES, ids=lambda d: "N{N}K{K}M{M}".format(**d))
@pytest.mark.parametrize("flux", [True, False], ids=["flux", "noflux"])
def test_step_matches_oracle(dims, flux):
    cfgd = _cfg(dict(dims, const_flux=flux))
    o, g = oracle_pipe(cfgd), device_pipe(cfgd)
    o.vel_matrices()
    g.vel_matrices()
    st = O.seeded_state(o, 21, 1e-3)
    o.set_state(*st)
    state_to_dev(g, st)
    for p in (o, g):
        p.vel_imposesym()
        p.vel_transform()
        p.vel_nonlinear()
        p.vel_predictor()
        for _ in range(2):
            p.vel_transform()
            p.vel_nonlinear()
            p.vel_corrector()
    tol = 1e-12 * max(1.0, (cfgd["N"] / 64) ** 4)
    assert O.rel_l2(state_from_dev(g), o.state()) <= tol
    # the largest correction comes back from the pipe's last tile
    assert abs(g.tim.dterr - o.tim_dterr) <= 1e-9 * o.tim_dterr
    g.close()


def test_step_in_a_batch_equals_alone():
    """Every launch shape, part-filled tiles of both kinds, and lone grids on
    either side of the SM count, in one batch of ten pipes."""
    import pipeflow as P
    cfgs = [P.PipeConfig(**_cfg(d)) for d in SIZES if 3 * d["K"] in (12, 15, 24, 48) and 3 * d["M"] in (12, 15, 18)]
    cfgs += [P.PipeConfig(**_cfg(dict(N=N, K=64, M=32))) for N in (20, 40, 56)]  # larger than the GPU
    cfgs += [P.PipeConfig(**_cfg(dict(N=64, K=4, M=4, Re=1900.0)))]  # pivots in the Helmholtz factors
    batch = P.Batch(cfgs)
    batch.matrices()
    alone = [P.Pipe(c) for c in cfgs]
    for i, (b, a) in enumerate(zip(batch.pipes, alone)):
        a.vel_matrices()
        P.seeded_state(a, 60 + i, 1e-3)
        b.set_state(*a.get_state())
    batch.step(3)
    assert batch.staged()
    for b, a in zip(batch.pipes, alone):
        for _ in range(3):
            a.timestep()
        for (br, bi), (ar, ai) in zip(b.get_state(), a.get_state()):
            assert np.array_equal(br, ar) and np.array_equal(bi, ai)
        a.close()
    batch.close()
