"""Passes that a rule sends to the register kernels are not slower there than in the tiled kernel (GPU)."""
import numpy as np
import pytest

from decomp_mpi_gb300 import api

pytestmark = pytest.mark.gpu
ARITH = {"fp64": (api.C128, api.ARITH_FP64), "fp32": (api.C64, api.ARITH_FP32), "df": (api.C128, api.ARITH_DF)}


def _microseconds(run, cuda):
    import torch
    stream = torch.cuda.current_stream().cuda_stream
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)

    def once(reps):
        torch.cuda.synchronize()
        a.record()
        for _ in range(reps):
            run(stream)
        b.record()
        torch.cuda.synchronize()
        return a.elapsed_time(b) * 1e3 / reps

    once(1)
    reps = 20 if once(1) < 2e3 else 2
    return min(once(reps) for _ in range(7))


def _plan(cuda, spec, shape, name):
    import torch
    dtype, arith = ARITH[name]
    comm = api.Comm(1)
    S = api.decomp_from_spec(comm, spec)
    n = int(np.prod(shape))
    cd = torch.complex128 if dtype == api.C128 else torch.complex64
    dat, work = torch.randn(n, dtype=cd, device=cuda), torch.zeros(2 * n, dtype=cd, device=cuda)
    plan = api.SplitPlan(S, dat.data_ptr(), 2 * n, work.data_ptr(), dtype=dtype, arith=arith)
    plan.keep = (comm, S, dat, work)
    return plan


def _not_slower(cuda, spec, shape, name):
    """Against the same plan with the tiled kernel's own tile; 10 % and 1 us for the spread of the timing."""
    plan = _plan(cuda, spec, shape, name)
    tiled = _plan(cuda, spec, shape, name)
    tiled.set_tile({"fp64": 1024, "df": 2048, "fp32": 4096}[name])
    for d in (api.FFTW_FORWARD, api.FFTW_BACKWARD):
        now, was = (_microseconds(lambda s: p.run(d, s), cuda) for p in (plan, tiled))
        assert now <= 1.1 * was + 1.0, (shape, name, now, was, plan.describe())


@pytest.mark.parametrize("name", list(ARITH))
@pytest.mark.parametrize("shape", [(211,), (13,), (37, 64), (211, 48), (48, 211), (66, 66, 66)], ids=str)
def test_direct_primes(shape, name, cuda):
    _not_slower(cuda, "packed:" + "|".join("local(%d)" % n for n in shape), shape, name)



@pytest.mark.parametrize("name", list(ARITH))
@pytest.mark.parametrize("shape", [(1331, 512), (512, 1331), (143, 1024)], ids=str)
def test_twiddled_primes(shape, name, cuda):
    _not_slower(cuda, "packed:" + "|".join("local(%d)" % n for n in shape), shape, name)



@pytest.mark.parametrize("name", list(ARITH))
@pytest.mark.parametrize("shape", [(720, 512), (600, 512), (1000, 512), (1536, 512), (512, 1280), (1000, 64)], ids=str)
def test_lines_for_part_of_the_chip(shape, name, cuda):
    """As many blocks of any-length lines as SMs, or a few times that."""
    _not_slower(cuda, "packed:" + "|".join("local(%d)" % n for n in shape), shape, name)



@pytest.mark.parametrize("name", list(ARITH))
@pytest.mark.parametrize("shape", [(7, 1024), (1024, 64), (128, 1024), (1024, 300)], ids=str)
def test_few_long_lines(shape, name, cuda):
    _not_slower(cuda, "packed:" + "|".join("local(%d)" % n for n in shape), shape, name)



@pytest.mark.parametrize("name", list(ARITH))
@pytest.mark.parametrize("spec,shape", [("packed:local(2048)|local(1024)", (2048, 1024)),
                                        ("packed:local(512)|local(2048)", (512, 2048)),
                                        ("packed:local(2048)|local(64)", (2048, 64))], ids=lambda v: str(v)[:40])
def test_lengths_without_a_schedule(spec, shape, name, cuda):
    _not_slower(cuda, spec, shape, name)
