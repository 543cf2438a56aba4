"""A further corrector pass of part of a batch whose mixed-precision transforms
run one block per radial point: the masked launches of that kernel against the
same pipes stepped alone on the three passes, bit for bit.
"""
import numpy as np
import pytest

from test_gpu_batch_corrector import AMP, DTERR

pytestmark = pytest.mark.gpu

BASE = dict(Mp=1, Re=2200.0, alpha=1.1, dt=0.01)
# three shapes that have the one-block kernel, one whose plane does not fit, one FP64 pipe
PIPES = [(32, 16, 12, True), (24, 32, 24, True), (40, 24, 16, True), (16, 64, 24, True), (24, 6, 5, False)]


@pytest.mark.parametrize("graphs", [True, False], ids=["graphs", "direct"])
def test_masked_pass_of_one_block_transforms(graphs):
    import pipeflow as P
    cfgs = [P.PipeConfig(N=N, K=K, M=M, **BASE, precision=P.PF_PREC_MIXED if mx else P.PF_PREC_FP64, dterr=e)
            for (N, K, M, mx), e in zip(PIPES, DTERR)]
    batch = P.Batch(cfgs)
    batch.set_graphs(graphs)
    batch.matrices()
    alone = [P.Pipe(c) for c in cfgs]
    for i, (b, a) in enumerate(zip(batch.pipes, alone)):
        b.set_tuning(nl_fused=1)
        a.vel_matrices()
        P.seeded_state(b, 100 + i, AMP[i])
        P.seeded_state(a, 100 + i, AMP[i])
    assert [b.nl_passes for b in batch.pipes] == [1, 1, 1, 3, 3]
    passes = batch.step(4)
    n = [[a.timestep() for _ in range(4)] for a in alone]
    assert passes == sum(map(sum, n))
    assert len({k[-1] for k in n}) >= 2, n
    for b, a in zip(batch.pipes, alone):
        for (br, bi), (ar, ai) in zip(b.get_state(), a.get_state()):
            assert np.array_equal(br, ar) and np.array_equal(bi, ai)
        a.close()
    batch.close()
