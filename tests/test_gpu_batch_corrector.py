"""Further corrector passes of part of a batch.

The pipes that have not converged take their next pass together, the others
are left alone: state, step control and the number of passes must equal the
same pipes stepped alone, bit for bit.
"""
import numpy as np
import pytest

from test_gpu_batch import PIVOTING, UNEVEN

pytestmark = pytest.mark.gpu

DTERR = (1e-5, 1e-8, 1e-6, 1e-8, 1e-7)  # one to six passes
AMP = (1e-3, 2e-1, 3e-2, 1e-2, 1e-1)
MIRROR = dict(N=32, K=8, M=8, Mp=1, Re=2000.0, alpha=1.0, dt=0.01, mirrorsym=True)

# (precision of each pipe, last pipe, graphs, one launch per transform pass)
VARIANTS = {
    "fp64": ((0, 0, 0, 0, 0), PIVOTING, True, False),
    "uneven": ((1, 0, 0, 1, 1), PIVOTING, True, False),
    "mixed-worklist": ((1, 1, 1, 1, 1), PIVOTING, True, True),
    "direct": ((0, 1, 1, 0, 1), PIVOTING, False, False),
    "branch": ((0, 0, 0, 0, 0), MIRROR, True, False),
}


@pytest.mark.parametrize("variant", list(VARIANTS))
def test_corrector_passes_of_part_of_a_batch(variant):
    import pipeflow as P
    prec, last, graphs, worklist = VARIANTS[variant]
    cfgs = [P.PipeConfig(**d, precision=q, dterr=e) for d, q, e in zip(UNEVEN + [last], prec, DTERR)]
    batch = P.Batch(cfgs)
    batch.set_graphs(graphs)
    batch.set_worklist(worklist)
    batch.matrices()
    alone = [P.Pipe(c) for c in cfgs]
    for i, (b, a) in enumerate(zip(batch.pipes, alone)):
        a.vel_matrices()
        P.seeded_state(b, 100 + i, AMP[i])
        P.seeded_state(a, 100 + i, AMP[i])
    nsteps = 4  # both parities of the recorded pass, twice with one state in the first step
    passes = batch.step(nsteps)
    assert batch.staged() == (last is PIVOTING)
    n = [[a.timestep() for _ in range(nsteps)] for a in alone]
    assert passes == sum(map(sum, n))
    assert len({k[-1] for k in n}) >= 3, n
    for b, a in zip(batch.pipes, alone):
        for (br, bi), (ar, ai) in zip(b.get_state(), a.get_state()):
            assert np.array_equal(br, ar) and np.array_equal(bi, ai)
        for f in ("t", "step", "it", "dt", "dterr", "corr_dt"):
            assert getattr(b.tim, f) == getattr(a.tim, f), f
    batch.close()
