"""Grouped runs whose passes go to two kernels: the register kernel of any length, and the tiled kernel's runtime stages
for the passes it does not take (here a plan with a tile size of the caller's, and ranked sides in the split schedule)."""
import ctypes

import numpy as np
import pytest

from decomp_mpi_gb300 import api
from decomp_mpi_gb300._lib import load
from oracle import oracle as O

# (ranks, start decomposition, shape, schedule, tile)
GROUP = [
    (4, "packed:block(32,2)|block(24,2)|local(20)", (32, 24, 20), api.SCHEDULE_LINES, 0),
    (6, "packed:block(50,3)|block(36,2)", (50, 36), api.SCHEDULE_LINES, 64),
    (8, "packed:block(14,2)|block(21,4)|local(11)", (14, 21, 11), api.SCHEDULE_SPLIT, 0),
]
ARITH = {"fp64": (api.C128, api.ARITH_FP64), "df": (api.C128, api.ARITH_DF), "fp32": (api.C64, api.ARITH_FP32)}
TILED = 0


def _plan(job, name, dat, work):
    P, spec, shape, schedule, tile = job
    dtype, arith = ARITH[name]
    comm = api.Comm(P)
    S = api.decomp_from_spec(comm, spec)
    plan = api.SplitPlan(S, dat, 2 * int(np.prod(shape)), work, dtype=dtype, arith=arith, schedule=schedule)
    plan.set_radix(api.RADIX_PLAN8)
    plan.set_tile(tile)
    plan.keep = (comm, S)
    return plan


def _forms(plan, direction):
    out = (ctypes.c_int * 16)()
    fn = load().dmg_split_pass_forms
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int)]
    return list(out[:fn(plan.h, direction, 0, out)])


@pytest.mark.parametrize("name", list(ARITH))
@pytest.mark.parametrize("which", [(0,), (1,), (0, 1), (0, 2), (0, 1, 2)], ids=str)
def test_launches_are_counted_per_kernel(which, name):
    plans = [_plan(GROUP[i], name, 1 << 20, 1 << 24) for i in which]
    for d in (api.FFTW_FORWARD, api.FFTW_BACKWARD):
        forms = [_forms(p, d) for p in plans]
        assert all(f == TILED for f in forms[which.index(1)]) if 1 in which else True
        kernels = [{f[k] == TILED for f in forms if k < len(f)} for k in range(max(map(len, forms)))]
        pre = len(plans) if name == "df" else 0
        assert api.split_group_launches(plans, d) == sum(map(len, kernels)) + pre
    if set(which) == {0, 1}:
        assert {True, False} in kernels  # (both kernels in one pass index)


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(ARITH))
def test_results_are_the_plans_own(name, cuda):
    """The same bits as each plan's own run; a line of infinities and NaN in one array leaves the others alone."""
    import torch
    tdt = torch.complex128 if name != "fp32" else torch.complex64
    stream = torch.cuda.current_stream(cuda).cuda_stream
    plans, host, dat, work, globs = [], [], [], [], []
    for i, job in enumerate(GROUP):
        P, spec, shape = job[:3]
        S = api.decomp_from_spec(api.Comm(P), spec)
        rng = np.random.default_rng(40 + i)
        glob = rng.uniform(-1, 1, shape) + 1j * rng.uniform(-1, 1, shape)
        globs.append(glob)
        host.append(torch.from_numpy(O.scatter_global(P, spec, glob, S.extent())).to(tdt))
        dat.append(host[i].to(cuda))
        work.append(torch.zeros(P * 2 * int(np.prod(shape)), dtype=tdt, device=cuda))
        plans.append(_plan(job, name, dat[i].data_ptr(), work[i].data_ptr()))
    own = []
    for p, w in zip(plans, work):
        p.run(api.FFTW_FORWARD, stream)
        torch.cuda.synchronize()
        own.append(torch.view_as_real(w).clone())

    def grouped():
        for w in work:
            w.zero_()
        api.split_run_group(plans, api.FFTW_FORWARD, stream)
        torch.cuda.synchronize()

    grouped()
    for w, o in zip(work, own):
        assert torch.equal(torch.view_as_real(w), o)
    if name != "df":  # (double-float scales by the largest value, which has to be finite)
        dat[0].copy_(host[0])
        dat[0][:20] = complex(float("inf"), float("nan"))
        grouped()
        # (every value of the spectrum's layout; the rest of the workspace holds passes in between)
        _, mask = O.split_expected_output(*GROUP[0][:2], globs[0], 2 * globs[0].size)
        assert not np.isfinite(torch.view_as_real(work[0]).cpu().numpy()[mask]).any()
        for w, o in zip(work[1:], own[1:]):
            assert torch.equal(torch.view_as_real(w), o)
