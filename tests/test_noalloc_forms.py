"""Which kernels dmg_split_run_noalloc's passes take (CPU): those of the regular run, at every workspace pitch.

Its intermediate sides lie in the fixed scratch array, whose rank pitch is the dense extent.  A workspace pitch that puts
offsets along a line beyond 32 bits keeps the regular pass out of the register kernels; the scratch pass then stays out
too, since their twiddle tables are made for the regular pass and both runs give the same bits."""
import ctypes

import pytest

from decomp_mpi_gb300 import api
from decomp_mpi_gb300._lib import load

TILED = 0


def _forms(plan, direction, noalloc):
    out = (ctypes.c_int * 16)()
    fn = load().dmg_split_pass_forms
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int)]
    return list(out[:fn(plan.h, direction, noalloc, out)])


@pytest.mark.parametrize("length", [None, 1 << 31, 1 << 40], ids=["dense", "2^31", "2^40"])
@pytest.mark.parametrize("dtype,arith", [(api.C128, api.ARITH_FP64), (api.C128, api.ARITH_DF), (api.C64, api.ARITH_FP32)],
                         ids=["fp64", "df", "fp32"])
@pytest.mark.parametrize("P,spec,schedule", [
    (4, "packed:block(64,2)|block(64,2)", api.SCHEDULE_LINES),   # two passes: one intermediate, in the upper half
    (4, "packed:block(64,2)|block(50,2)", api.SCHEDULE_LINES),   # the kernel of any length
    (6, "packed:block(64,3)|block(48,2)", api.SCHEDULE_LINES),   # ranked sides
    (4, "packed:block(1024,2)|block(64,2)|local(16)", api.SCHEDULE_SPLIT),
    (4, "packed:block(32,2)|block(48,2)|local(64)", api.SCHEDULE_LINES),
])
def test_scratch_passes_take_the_regular_forms(P, spec, schedule, dtype, arith, length):
    comm = api.Comm(P)
    start = api.decomp_from_spec(comm, spec)
    wl = length or 2 * api.SplitPlan(start, 1 << 20, 1 << 40, 1 << 21, dtype=dtype).extent64
    plan = api.SplitPlan(start, 1 << 20, wl, 1 << 21, dtype=dtype, arith=arith, schedule=schedule)
    for d in (api.FFTW_FORWARD, api.FFTW_BACKWARD):
        regular = _forms(plan, d, 0)
        assert _forms(plan, d, 1) == regular
        if length is not None and schedule == api.SCHEDULE_LINES and P == 4:
            assert TILED in regular  # (the pitch does keep a pass out of the register kernels)
