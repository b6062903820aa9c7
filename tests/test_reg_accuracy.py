"""How far results are from exact ones (longer arithmetic on the host), kernel against kernel: what the oracle tests'
tolerances, some thirty times the errors, do not see."""
import numpy as np
import pytest

from decomp_mpi_gb300 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu
LONG = np.finfo(np.longdouble).eps < 2.0 ** -60


def _arrays(n, along_t):
    """Random arrays of lines of n points, 2 lines each (two points along the other dimension: one exact stage)."""
    shape = (2, n) if along_t else (n, 2)
    rng = np.random.default_rng(n)
    count = max(4, 65536 // n)
    return shape, [rng.uniform(-1, 1, shape) + 1j * rng.uniform(-1, 1, shape) for _ in range(count)]


def _errors(cuda, arrays, shape, dtype, arith, setups):
    """Relative L2 error of forward transforms over all arrays, per setup (a function that prepares the plan)."""
    import torch
    spec = "packed:" + "|".join("local(%d)" % n for n in shape)
    comm = api.Comm(1)
    S = api.decomp_from_spec(comm, spec)
    A, B, _, _, a_spec, b_spec = O.split_factors(1, spec)
    size = int(np.prod(shape))
    work = torch.zeros(2 * size, dtype=torch.complex128 if dtype == api.C128 else torch.complex64, device=cuda)
    off = O.global_offsets(1, a_spec if all(a == 1 for a in A) else b_spec, 2 * size, shape).ravel()
    freq = np.ix_(*[np.arange(n) // a + b * (np.arange(n) % a) for n, a, b in zip(shape, A, B)])
    err, norm = np.zeros(len(setups)), 0.0
    plans = []
    for setup in setups:
        plan = api.SplitPlan(S, work.data_ptr(), 2 * size, work.data_ptr(), dtype=dtype, arith=arith,
                             schedule=api.SCHEDULE_LINES)
        setup(plan)
        plans.append(plan)
    for x in arrays:
        x = x if dtype == api.C128 else x.astype(np.complex64)
        dat = torch.from_numpy(x.reshape(-1)).to(cuda)
        exact = np.fft.fftn(x.astype(np.clongdouble))[freq].ravel()
        assert exact.dtype == np.clongdouble
        norm += float(np.sum(np.abs(exact) ** 2))
        for i, plan in enumerate(plans):
            plan.set_buffers(dat.data_ptr(), work.data_ptr())
            plan.run(api.FFTW_FORWARD, torch.cuda.current_stream().cuda_stream)
            err[i] += float(np.sum(np.abs(work.cpu().numpy()[off] - exact) ** 2))
    return np.sqrt(err / norm), plans


@pytest.mark.skipif(not LONG, reason="no longer float on the host")
@pytest.mark.parametrize("along_t", [False, True], ids=["v1", "t"])
@pytest.mark.parametrize("n,radix", [(20, api.RADIX_FIXED), (72, api.RADIX_FIXED), (576, api.RADIX_FIXED),
                                     (32, api.RADIX_PLAN8), (768, api.RADIX_PLAN8), (256, api.RADIX_PLAN4)])
def test_any_length_fp64_is_no_further_off_than_the_tiled_kernel(n, radix, along_t, cuda):
    """Twiddled radix 8 and 4 in native FP64.  Both kernels round each twiddle product and each butterfly addition
    once, so their errors agree up to the sampling of about 65536 independent values (a relative 0.3 % in the root
    mean square) and the order of the radices; 3 % covers ten times the former."""
    shape, arrays = _arrays(n, along_t)
    err, plans = _errors(cuda, arrays, shape, api.C128, api.ARITH_FP64,
                         [lambda p: p.set_radix(radix), lambda p: (p.set_radix(radix), p.set_tile(1024))])
    assert "regs=any" in plans[0].describe() and "regs" not in plans[1].describe()
    assert err[0] <= 1.03 * err[1], err
