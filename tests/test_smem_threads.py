"""Plans of one kernel with different shared memory, launched from several host threads at once (GPU).

The limit on a kernel's dynamic shared memory belongs to the function, not to the launch: a thread that lowered it
between another thread's raising it and its launch would have that launch refused."""
import threading

import numpy as np
import pytest

from decomp_mpi_gb300 import api

pytestmark = pytest.mark.gpu
ROUNDS = 4000


def _race(cuda, runs):
    import torch
    errors = []
    go = threading.Barrier(len(runs))

    def work(run):
        torch.cuda.set_device(cuda)
        stream = torch.cuda.Stream(cuda)
        go.wait()
        try:
            for k in range(ROUNDS):
                run(stream.cuda_stream)
                if k % 100 == 99:
                    stream.synchronize()
        except Exception as e:  # a refused launch
            errors.append(e)
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(r,)) for r in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors


@pytest.mark.parametrize("lengths,radix", [((1000, 360), api.RADIX_FIXED), ((1024, 144), api.RADIX_PLAN8)],
                         ids=["any length", "plan radices"])
def test_fft_passes(lengths, radix, cuda):
    import torch
    keep, want, runs = [], [], []
    for n in lengths:
        comm = api.Comm(1)
        S = api.decomp_from_spec(comm, "packed:local(%d)|local(64)" % n)
        rng = np.random.default_rng(n)
        x = rng.uniform(-1, 1, 64 * n) + 1j * rng.uniform(-1, 1, 64 * n)
        dat = torch.from_numpy(x).to(cuda)
        work = torch.zeros(128 * n, dtype=torch.complex128, device=cuda)
        plan = api.SplitPlan(S, dat.data_ptr(), 128 * n, work.data_ptr(), dtype=api.C128, arith=api.ARITH_FP64)
        plan.set_radix(radix)
        plan.run(api.FFTW_FORWARD, torch.cuda.current_stream(cuda).cuda_stream)
        torch.cuda.synchronize()
        want.append(work.clone())
        keep.append((comm, S, dat, work, plan))
        runs.append(lambda s, p=plan: p.run(api.FFTW_FORWARD, s))
    _race(cuda, runs)
    for w, k in zip(want, keep):
        assert torch.equal(torch.view_as_real(w), torch.view_as_real(k[3]))


def test_ranked_reshapes(cuda):
    import torch
    comm = api.Comm(64)
    keep, runs = [], []
    # (short rows and many positions: tables of 26 and 32 KB, two per block)
    for src, dst in (("packed:local(60)|block(41,21)", "packed:local(60)|block(41,20)"),
                     ("packed:local(64)|block(41,17)", "packed:local(64)|block(41,16)")):
        plan = api.ReshapePlan(comm, 16, api.decomp_from_spec(comm, src), api.decomp_from_spec(comm, dst))
        a = torch.zeros(64 * plan.src_pitch * 16, dtype=torch.uint8, device=cuda)
        b = torch.zeros(64 * plan.dest_pitch * 16, dtype=torch.uint8, device=cuda)
        keep.append((plan, a, b))
        runs.append(lambda s, p=plan, a=a, b=b: p.run(a.data_ptr(), b.data_ptr(), s))
    _race(cuda, runs)
