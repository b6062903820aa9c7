"""Register passes of few 1024-point lines, a line to a block, give the bits of the passes with the schedule's four (GPU):
a batch of more lines takes the latter, each of its arrays alone the former."""
import numpy as np
import pytest

from decomp_mpi_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith", [api.ARITH_FP64, api.ARITH_DF], ids=["fp64", "df"])
@pytest.mark.parametrize("shape", [(1024, 64), (64, 1024), (1024, 31), (31, 1024)], ids=str)
def test_alone_and_in_a_batch(shape, arith, cuda):
    import torch
    jobs, n = 16, int(np.prod(shape))
    comm = api.Comm(1)
    S = api.decomp_from_spec(comm, "packed:local(%d)|local(%d)" % shape)
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (jobs, n)) + 1j * rng.uniform(-1, 1, (jobs, n))
    dat = torch.from_numpy(x).to(cuda)
    work = torch.zeros((jobs, 2 * n), dtype=torch.complex128, device=cuda)
    scales = torch.zeros(jobs, dtype=torch.int32, device=cuda)
    stream = torch.cuda.current_stream(cuda).cuda_stream
    plan = api.SplitPlan(S, dat.data_ptr(), 2 * n, work.data_ptr(), dtype=api.C128, arith=arith,
                         schedule=api.SCHEDULE_LINES)
    assert "n=1024" in plan.describe() and "regs=" in plan.describe()
    for d, result in ((api.FFTW_FORWARD, work), (api.FFTW_BACKWARD, dat)):
        source = (dat if d == api.FFTW_FORWARD else work).clone()
        plan.run_batch(d, [dat[j].data_ptr() for j in range(jobs)], [work[j].data_ptr() for j in range(jobs)],
                       scales=[scales[j:].data_ptr() for j in range(jobs)], stream=stream)
        torch.cuda.synchronize()
        batch = torch.view_as_real(result).clone()
        (dat if d == api.FFTW_FORWARD else work).copy_(source)
        result.zero_()
        for j in range(jobs):
            plan.set_buffers(dat[j].data_ptr(), work[j].data_ptr())
            plan.run(d, stream)
        torch.cuda.synchronize()
        assert torch.equal(torch.view_as_real(result), batch)
    assert np.abs(dat.cpu().numpy() / n - x).max() < 1e-12
