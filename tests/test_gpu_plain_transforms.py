"""The plain transforms (coll to phys and back, one and several fields, and the
allocation-free one) against the oracle's at every compiled length and at
lengths of each radix, with a radial size that no tile divides, part-filled z
tiles and a single mode.  Tolerance: the repository's bar for a transform."""
import ctypes as C

import numpy as np
import pytest

from _util import device_pipe, from_dev, oracle_pipe, rand_coll, rel, rel_coll, to_dev

pytestmark = pytest.mark.gpu
TOL = 1e-13

# 3K and 3M: each of 12 15 18 24 36 48 72 96 144 192 288 384 in both places
COMPILED = [(4, 128), (5, 96), (6, 64), (8, 48), (12, 32), (16, 24), (24, 16), (32, 12), (48, 8), (64, 6), (96, 5),
            (128, 4)]
# radices 2 3 4 5 7 11 13, odd and even lengths, mixed with compiled ones
GENERIC = [(1, 1), (2, 7), (7, 2), (11, 13), (13, 11), (20, 11), (35, 3), (22, 26), (3, 16), (24, 21), (70, 9)]


@pytest.mark.parametrize("km", COMPILED + GENERIC, ids=lambda p: "K%dM%d" % p)
def test_plain_transforms(km):
    K, M = km
    cfgd = dict(N=11, K=K, M=M, Mp=1, Re=2000.0, alpha=1.25, dt=0.01)
    o, g = oracle_pipe(cfgd), device_pipe(cfgd)
    rng = np.random.default_rng(5)
    c = rand_coll(o.N, o.H, rng)
    ref = o.tra_spec2phys(c)
    p = g.phys()
    g.tra_coll2phys(to_dev(g, c), p)
    assert rel(p.download(), ref) < TOL
    phys = rng.standard_normal((o.N, o.cfg.Th, o.cfg.Z))
    out = g.coll()
    g.tra_phys2coll(g.phys(phys), out)
    assert rel_coll(from_dev(out), o.tra_phys2spec(phys)) < TOL
    if km in COMPILED:
        import torch
        d_re, d_im = (torch.from_numpy(np.ascontiguousarray(x.T)).to("cuda") for x in (c.re, c.im))
        got = torch.full((ref.size,), float("nan"), dtype=torch.float64, device="cuda")
        st = torch.cuda.current_stream().cuda_stream
        ok = g.lib.pf_tra_coll2phys_noalloc(11, K, M, *(C.c_void_p(x.data_ptr()) for x in (d_re, d_im, got)),
                                            C.c_void_p(st))
        torch.cuda.synchronize()
        assert ok == 0 and rel(got.cpu().numpy().reshape(ref.shape), ref) < TOL
