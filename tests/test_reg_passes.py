"""Passes whose butterflies run in registers (fft_reg.cuh: lengths with a compile-time schedule; fft_gen.cuh: any
length, ranked sides, groups): which passes take which form (CPU), and every length, arithmetic and form against
the FP64 oracle and the tiled kernel (GPU)."""
import re

import numpy as np
import pytest

from decomp_mpi_gb300 import api
from oracle import oracle as O

LENGTHS = (32, 48, 64, 96, 120, 128, 160, 192, 240, 256, 320, 384, 480, 512, 1024, 2048)
# relative L2 error of a transform of N values: 8 u log2 N, u the unit roundoff of the arithmetic (double-float:
# 48-bit significands whose operations lose up to two bits)
UNIT = {"fp64": 2.0 ** -53, "fp32": 2.0 ** -24, "df": 2.0 ** -46}
ARITH = {"fp64": (api.C128, api.ARITH_FP64), "fp32": (api.C64, api.ARITH_FP32), "df": (api.C128, api.ARITH_DF)}


def _forms(plan):
    return re.findall(r"n=(\d+) [^\]]*? tiles=\d+(?: slots| tw)?(?: regs=(\w+))? in=", plan.describe())


def _plan(P, spec, **kw):
    comm = api.Comm(P)
    start = api.decomp_from_spec(comm, spec)
    probe = api.SplitPlan(start, 1 << 20, 1 << 40, 1 << 21, dtype=kw.get("dtype", api.C128))
    return api.SplitPlan(start, 1 << 20, 2 * probe.extent64, 1 << 21, **kw)


def test_which_passes_keep_lines_in_registers():
    even = "packed:block(64,2)|block(48,2)|local(128)"
    p = _plan(4, even)
    assert _forms(p) == [("128", "t"), ("48", "v1"), ("64", "v1")]
    p.set_tile(1024)  # an explicit tile size keeps the tiled kernel
    assert [f for _, f in _forms(p)] == ["", "", ""]
    p.set_tile(0)
    p.set_radix(api.RADIX_PLAN8)  # the caller's radices run in the kernel of any length
    assert [f for _, f in _forms(p)] == ["any", "any", "any"]
    p.set_radix(api.RADIX_FIXED)
    # rank buffers too far apart for 32-bit offsets along the line
    far = api.SplitPlan(p.start, 1 << 20, 1 << 40, 1 << 21)
    assert _forms(far) == [("128", ""), ("48", "v1"), ("64", "v1")]
    # a length without a schedule; 2048 points for 8-byte values only (the first double-float pass converts, which
    # keeps lengths with compile-time tiled stages there unless both sides are ranked)
    assert _forms(_plan(4, "packed:block(64,2)|block(50,2)|local(128)")) == [("128", "t"), ("50", "any"), ("64", "v1")]
    for dtype, form in ((api.C64, "t"), (api.C128, "")):
        assert _forms(_plan(4, "packed:block(8,2)|block(8,2)|local(2048)", dtype=dtype,
                            schedule=api.SCHEDULE_LINES))[0] == ("2048", form)
    # the tensor-core form keeps its own 1024-point kernel
    assert _forms(_plan(4, "packed:block(32,2)|block(32,2)|local(1024)", dtype=api.C64,
                        arith=api.ARITH_TC16)) == [("1024", ""), ("32", "v1"), ("32", "v1")]
    # uneven blocks: per-rank strides on the start side
    assert _forms(_plan(12, "packed:block(64,3)|block(48,4)|local(128)"))[:2] == [("128", ""), ("48", "any")]
    # Fortran order in memory: the first pass reads along v2 or v1 and writes along t
    fortran = "axes:block(64,2)@1,1|block(64,2)@32,2|local(64)@1024,4"
    assert _forms(_plan(4, fortran))[0] == ("64", "")
    assert _forms(_plan(4, fortran, dtype=api.C64))[0] == ("64", "any")
    # the split schedule: an interleaved layout's lines share their offsets
    s = _plan(4, "packed:block(1024,2)|block(64,2)|local(64)", schedule=api.SCHEDULE_SPLIT)
    assert ("32", "v1") in _forms(s), s.describe()


def _run(cuda, P, spec, shape, name, seed, **kw):
    import torch
    dtype, arith = ARITH[name]
    comm = api.Comm(P)
    S = api.decomp_from_spec(comm, spec)
    rng = np.random.default_rng(seed)
    glob = rng.uniform(-1, 1, shape) + 1j * rng.uniform(-1, 1, shape)
    if dtype == api.C64:
        glob = glob.astype(np.complex64).astype(np.complex128)
    host = O.scatter_global(P, spec, glob, S.extent()).astype(np.complex128 if dtype == api.C128 else np.complex64)
    dat = torch.from_numpy(host).to(cuda)
    probe = api.SplitPlan(S, 1 << 20, 1 << 40, 1 << 21, dtype=dtype)
    wl = 2 * probe.extent64
    work = torch.zeros(P * wl, dtype=dat.dtype, device=cuda)
    plan = api.SplitPlan(S, dat.data_ptr(), wl, work.data_ptr(), dtype=dtype, arith=arith, **kw)
    return plan, dat, work, glob, S.extent(), wl


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(ARITH))
@pytest.mark.parametrize("n", LENGTHS)
def test_length_against_the_oracle(n, name, cuda):
    """Line counts that leave the last block of lines partly empty, in both forms, forward and back."""
    import torch
    if n == 2048 and name != "fp32":
        pytest.skip("no register schedule")
    for P, spec, shape in ((1, "packed:local(3)|local(7)|local(%d)" % n, (3, 7, n)),
                           (2, "packed:local(%d)|block(6,2)|local(7)" % n, (n, 6, 7)),
                           (2, "packed:block(4,2)|local(%d)|local(5)" % n, (4, n, 5))):
        plan, dat, work, glob, pitch, wl = _run(cuda, P, spec, shape, name, n)
        assert (str(n), "t" if shape[2] == n else "v1") in _forms(plan), plan.describe()
        tol = 8 * UNIT[name] * np.log2(np.prod(shape))
        plan.run(api.FFTW_FORWARD, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        exp, mask = O.split_expected_output(P, spec, glob, wl)
        assert _rel(work.cpu().numpy()[mask].astype(np.complex128), exp[mask]) < tol, shape
        plan.run(api.FFTW_BACKWARD, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        back = O.gather_global(P, spec, dat.cpu().numpy().astype(np.complex128), pitch, shape) / np.prod(shape)
        assert _rel(back, glob) < 2 * tol, shape


LAYOUTS = [
    # start layouts that reorder the lines: rotated, reversed factors, interleaved, and both passes of a
    # dimension in the split schedule (twiddles after the transform forward, before it inverse)
    (8, "packed:frev(8,8,block(64,4))|rotate(5,block(48,2))|local(32)", (64, 48, 32), None),
    (4, "packed:interleave(block(16,2),4)|frev(6,8,block(48,2))|local(96)", (64, 48, 96), None),
    (4, "packed:local(32)|block(64,2)|block(48,2)", (32, 64, 48), None),
    (8, "packed:block(1024,4)|block(64,2)|local(96)", (1024, 64, 96), api.SCHEDULE_SPLIT),
    (4, "packed:block(4096,2)|block(64,2)|local(48)", (4096, 64, 48), api.SCHEDULE_SPLIT),
]


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(ARITH))
@pytest.mark.parametrize("P,spec,shape,schedule", LAYOUTS, ids=[str(c[2]) for c in LAYOUTS])
def test_layouts_against_the_tiled_kernel(P, spec, shape, schedule, name, cuda):
    """The same slots of the workspace and of dat as the tiled kernel (an explicit tile size), every slot."""
    import torch
    out = []
    for tile in (0, 1024):
        plan, dat, work, glob, pitch, wl = _run(cuda, P, spec, shape, name, 3, schedule=schedule)
        plan.set_tile(tile)
        assert any(f for _, f in _forms(plan)) == (tile == 0), plan.describe()
        st = torch.cuda.current_stream().cuda_stream
        plan.run(api.FFTW_FORWARD, st)
        torch.cuda.synchronize()
        spectrum = work.cpu().numpy().astype(np.complex128)
        plan.run(api.FFTW_BACKWARD, st)
        torch.cuda.synchronize()
        out.append((spectrum, dat.cpu().numpy().astype(np.complex128)))
    _, mask = O.split_expected_output(P, spec, glob, wl)
    tol = 16 * UNIT[name] * np.log2(np.prod(shape))
    assert _rel(out[0][0][mask], out[1][0][mask]) < tol
    assert _rel(out[0][1], out[1][1]) < 2 * tol


ANY = [
    # (P, start spec, shape): single stages, composite radices, repeated primes, primes without a butterfly
    # alone, first and last; ranked sides (uneven blocks) on either side, along the lines and along t
    (1, "packed:local(7)|local(9)|local(2)", (7, 9, 2)),
    (2, "packed:block(14,2)|local(15)|local(10)", (14, 15, 10)),
    (4, "packed:block(25,2)|block(35,2)|local(63)", (25, 35, 63)),
    (6, "packed:block(45,3)|rotate(4,block(40,2))|local(105)", (45, 40, 105)),
    (7, "packed:local(13)|block(33,7)|local(37)", (13, 33, 37)),
    (12, "packed:block(30,4)|block(28,3)|local(128)", (30, 28, 128)),
    (5, "packed:block(243,5)|local(11)|local(6)", (243, 11, 6)),
    (4, "packed:local(6)|block(10,4)|local(1000)", (6, 10, 1000)),
    (4, "axes:block(64,2)@1,1|block(50,2)@32,2|local(36)@800,4", (64, 50, 36)),  # Fortran order in memory
    (3, "packed:block(343,3)", (343,)),
    (4, "packed:block(101,2)|block(26,2)", (101, 26)),
]


@pytest.mark.gpu
@pytest.mark.parametrize("radix", [api.RADIX_FIXED, api.RADIX_PLAN8], ids=["own", "plan8"])
@pytest.mark.parametrize("name", list(ARITH))
@pytest.mark.parametrize("P,spec,shape", ANY, ids=[str(c[2]) for c in ANY])
def test_any_length_against_the_oracle(P, spec, shape, name, radix, cuda):
    import torch
    plan, dat, work, glob, pitch, wl = _run(cuda, P, spec, shape, name, 5)
    plan.set_radix(radix)
    assert any(f == "any" for _, f in _forms(plan)), plan.describe()
    # (a direct prime DFT of p points sums p products one after the other)
    tol = 8 * UNIT[name] * (np.log2(np.prod(shape)) + max(q for n in shape for q in range(1, n + 1)
                                                          if n % q == 0 and all(q % r for r in range(2, q))))
    st = torch.cuda.current_stream().cuda_stream
    plan.run(api.FFTW_FORWARD, st)
    torch.cuda.synchronize()
    exp, mask = O.split_expected_output(P, spec, glob, wl)
    assert _rel(work.cpu().numpy()[mask].astype(np.complex128), exp[mask]) < tol
    plan.run(api.FFTW_BACKWARD, st)
    torch.cuda.synchronize()
    back = O.gather_global(P, spec, dat.cpu().numpy().astype(np.complex128), pitch, shape) / np.prod(shape)
    assert _rel(back, glob) < 2 * tol
