"""A fused step whose factor copies never arrived is its own pipe's failure.

The kernel reports it in the pipe's device scalars.  Here the report is written
there from the host, as the kernel would leave it, through a few lines built
against the library's own header: no copy is held back.  The wait itself is tried on
a barrier that nothing arrives at.
"""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from _util import SMALL, device_pipe

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
PLANT = r"""
#include "pf_internal.cuh"
extern "C" int plant(pf_ctx *c) {
    const int v = PF_STEP_STUCK;
    cudaStreamSynchronize(c->stream);
    return cudaMemcpy(&c->dsc->info, &v, sizeof(v), cudaMemcpyHostToDevice) == cudaSuccess ? 0 : 1;
}
// a barrier that nothing arrives at
static __global__ void k_wait(double *out) {
    __shared__ __align__(8) unsigned long long bar;
    const unsigned b = (unsigned)__cvta_generic_to_shared(&bar);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
    int tries = MBAR_TRIES;
    for (int i = 0; i < 2; ++i) {
        unsigned long long t0, t1;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0)::"memory");
        out[2 * i] = mbar_wait(b, 0, tries);
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1)::"memory");
        out[2 * i + 1] = (double)(t1 - t0) * 1e-9;
    }
}
extern "C" int wait_for_nothing(double *out) {
    double *d = nullptr;
    if (cudaMalloc((void **)&d, 32) != cudaSuccess) return 1;
    k_wait<<<1, 1>>>(d);
    const cudaError_t e = cudaMemcpy(out, d, 32, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def helper(tmp_path_factory):
    d = tmp_path_factory.mktemp("plant")
    (d / "plant.cu").write_text(PLANT)
    so = d / "plant.so"
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-shared", "-Xcompiler", "-fPIC", f"-I{ROOT / 'softx-d-17-00015_b200' / 'csrc'}", f"-I{ROOT / 'include'}", str(d / "plant.cu"),
                    "-o", str(so)], check=True)
    return C.CDLL(str(so))


@pytest.fixture
def plant(helper):
    helper.plant.argtypes = [C.c_void_p]
    return lambda ctx: helper.plant(ctx) == 0


def _state(cfgd, seed):
    import pipeflow as P
    p = device_pipe(cfgd)
    P.seeded_state(p, seed, 1e-3)
    st = p.get_state()
    p.close()
    return st


def _same(a, b):
    return all(np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1]) for x, y in zip(a, b))


def _status(fn):
    import pipeflow as P
    with pytest.raises(P.PipeflowError) as e:
        fn()
    return e.value.status


@pytest.mark.parametrize("last_aborts", [False, True])
@pytest.mark.parametrize("mirror", [False, True], ids=["staged", "branches"])
def test_a_batch_step_reports_it_whatever_the_other_pipes_report(plant, last_aborts, mirror):
    import pipeflow as P
    cfgs = [P.PipeConfig(**dict(SMALL[0], mirrorsym=mirror)) for _ in range(3)]
    batch = P.Batch(cfgs)
    batch.matrices()
    for i, p in enumerate(batch.pipes):
        P.seeded_state(p, 50 + i, 1e-3)
    batch.step(1)
    batch.step(1)
    if last_aborts:  # the corrector control's "dt --> 0" of the pipe after it
        t = batch.pipes[2].tim
        t.dt, t.step = 1e-10, 31
        batch.pipes[2].set_tim(t)
    assert plant(batch.pipes[1].ctx)
    dt, corr_dt = batch.pipes[1].tim.dt, batch.pipes[1].tim.corr_dt
    assert _status(lambda: batch.step(1)) == P._lib.PF_ERR_CUDA
    # the corrector control did not run on what the step left
    assert batch.pipes[1].tim.it == 0 and batch.pipes[1].tim.corr_dt == corr_dt and batch.pipes[1].tim.dt == dt
    batch.close()


def test_a_served_request_gets_it_and_the_others_their_results(plant):
    import pipeflow as P
    cfgd = SMALL[0]
    states = [_state(cfgd, 70 + i) for i in range(3)]
    srv = P.Server(hbm_budget=20 * 10**9, orbit=False)
    ids = [srv.submit(P.PipeConfig(**cfgd), 3, st) for st in states]
    srv.step()
    bh, ph = C.c_void_p(), C.c_void_p()
    assert srv.lib.pf_serve_batch(srv.h, C.byref(bh)) == 0 and srv.lib.pf_batch_pipe(bh, 1, C.byref(ph)) == 0
    assert plant(ph)
    assert _status(srv.step) == P._lib.PF_ERR_CUDA
    srv.step()
    assert set(srv.finished()) == set(ids)
    assert _status(lambda: srv.result(ids[1])) == P._lib.PF_ERR_CUDA
    for i in (0, 2):
        a = device_pipe(cfgd)
        a.vel_matrices()
        a.set_state(*states[i])
        for _ in range(3):
            a.timestep()
        assert _same(srv.result(ids[i]), a.get_state())
        a.close()
    # its memory serves the next request
    again = srv.submit(P.PipeConfig(**cfgd), 1, states[1])
    srv.step()
    srv.result(again)
    srv.close()


def test_new_matrices_start_a_pipe_afresh(plant):
    import pipeflow as P
    a, b = device_pipe(SMALL[2]), device_pipe(SMALL[2])
    st = _state(SMALL[2], 60)
    for p in (a, b):
        p.vel_matrices()
        p.set_state(*st)
    assert plant(a.ctx)
    assert _status(a.timestep) == P._lib.PF_ERR_CUDA
    assert _status(a.timestep) == P._lib.PF_ERR_CUDA  # the state is not to be trusted until then
    a.vel_matrices()
    a.set_state(*st)
    a.set_tim(b.tim)
    for p in (a, b):
        p.timestep()
    assert _same(a.get_state(), b.get_state())
    a.close()
    b.close()


def test_a_wait_gives_up_after_a_second_and_the_ones_after_it_at_once(helper):
    out = (C.c_double * 4)()
    assert helper.wait_for_nothing(out) == 0
    assert out[0] == 0.0 and 0.5 <= out[1] < 2.0
    assert out[2] == 0.0 and out[3] < 1e-3
