"""The largest z tiles that a tuning may ask for, and the next one up.

The cap of pf_ctx_set_tuning is 100 KiB for a tile of `nl_mc` transform rows
held as they were when the cap was drawn: two buffers of the FP64 rows of 3K =
288 and 384, else one buffer of padded rows, and two tables.
How a pass lays its rows out may change; which choices are taken may not, since
cached choices are set again without being timed.
"""
import numpy as np
import pytest

from _util import device_pipe

pytestmark = pytest.mark.gpu

# 3K, M, mixed, the largest nl_mc: (2 mc + 2) 3K 16 bytes, else rows of 24 x 17,
# 18 x 17, 16 x 13 and 16 x 13 elements: (row mc + 2 3K) 8 or 16 bytes
CAPS = [(384, 12, False, 7), (288, 12, False, 10), (384, 32, True, 29), (288, 48, True, 39), (192, 64, True, 59),
        (192, 32, False, 28)]


@pytest.mark.parametrize("Z,M,mixed,mc", CAPS, ids=lambda v: str(v))
def test_largest_z_tile_is_taken_and_the_next_is_not(Z, M, mixed, mc):
    import pipeflow as P
    cfgd = dict(N=10, K=Z // 3, M=M, Mp=1, Re=2200.0, alpha=1.1, dt=0.01)
    extra = {"precision": P.PF_PREC_MIXED} if mixed else {}
    a, b = device_pipe(cfgd, **extra), device_pipe(cfgd, **extra)
    for p in (a, b):
        p.vel_matrices()
    P.seeded_state(b, 4, 1e-3)
    a.set_state(*b.get_state())
    a.set_tuning(nl_mc=mc)
    for p in (a, b):
        p.timestep()
    for (ar, ai), (br, bi) in zip(a.get_state(), b.get_state()):
        assert np.array_equal(ar, br) and np.array_equal(ai, bi)
    with pytest.raises(P.PipeflowError) as e:
        a.set_tuning(nl_mc=mc + 1)
    assert e.value.status == P._lib.PF_ERR_ARG
    assert a.get_tuning()["nl_mc"] == mc
    a.close()
    b.close()
