"""GPU reshapes with ranked sides through the row tables (reshape_kernel.cu), bit for bit against the oracle."""
import numpy as np
import pytest

from decomp_mpi_gb300 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CASES = [
    # (P, src spec, dst spec, element bytes): several positions along the rows on one side or both, rows longer
    # than a tile, one-row tiles, one-value rows, coordinates a side does not hold, units of 1 to 16 bytes and more
    (35, "packed:local(50)|block(67,7)|block(38,5)", "packed:block(50,7)|block(67,5)|local(38)", 16),
    (35, "packed:block(50,7)|block(67,5)|local(38)", "packed:local(50)|block(67,7)|block(38,5)", 8),
    (12, "packed:block(31,3)|block(17,4)|local(9)", "packed:rotate(5,block(31,4))|block(17,3)|local(9)", 2),
    (6, "packed:block(5,2)|block(4100,3)", "packed:local(5)|block(4100,6)", 16),
    (12, "packed:block(7,2)|block(4100,6)", "packed:rotate(2,block(7,3))|rotate(9,block(4100,4))", 4),
    (10, "packed:block(11,5)|block(7,2)|local(1)", "packed:local(11)|block(7,3)|local(1)", 1),
    (9, "packed:block(10,3)|frev(4,5,block(20,3))|local(13)", "packed:block(10,9)|local(20)|local(13)", 48),
    (7, "packed:local(9)|block(40,7)|local(64)", "packed:block(9,2)|block(40,3)|local(64)", 16),
]


def _arrays(P, s_spec, d_spec, esize, cuda, seed):
    import torch
    comm = api.Comm(P)
    plan = api.ReshapePlan(comm, esize, api.decomp_from_spec(comm, s_spec), api.decomp_from_spec(comm, d_spec))
    rng = np.random.default_rng(seed)
    src = rng.integers(0, 256, (P * plan.src_pitch, esize), dtype=np.uint8)
    want = rng.integers(0, 256, (P * plan.dest_pitch, esize), dtype=np.uint8)
    dst = torch.from_numpy(want.copy()).to(cuda)
    vs, vw = (a.reshape(-1).view("V%d" % esize) for a in (src, want))
    O.reshape(P, s_spec, d_spec, vs, plan.src_pitch, vw, plan.dest_pitch)
    return plan, torch.from_numpy(src).to(cuda), dst, want


@pytest.mark.parametrize("P,s_spec,d_spec,esize", CASES)
def test_ranked_rows(P, s_spec, d_spec, esize, cuda):
    import torch
    plan, src, dst, want = _arrays(P, s_spec, d_spec, esize, cuda, 1)
    assert "ranked" in plan.describe()
    plan.run(src.data_ptr(), dst.data_ptr(), torch.cuda.current_stream(cuda).cuda_stream)
    torch.cuda.synchronize()
    assert np.array_equal(dst.cpu().numpy(), want)


def test_ranked_rows_grouped(cuda):
    """Ranked and separable moves of one unit size side by side in grouped launches."""
    import torch
    jobs = [_arrays(P, s, d, 16, cuda, k) for k, (P, s, d, _) in enumerate(CASES[:2] + CASES[6:])]
    jobs.append(_arrays(4, "packed:block(8,2)|block(6,2)|local(5)", "packed:local(8)|block(6,2)|block(5,2)", 16, cuda, 9))
    api.reshape_group([j[0] for j in jobs], [j[1].data_ptr() for j in jobs], [j[2].data_ptr() for j in jobs],
                      torch.cuda.current_stream(cuda).cuda_stream)
    torch.cuda.synchronize()
    for plan, _, dst, want in jobs:
        assert np.array_equal(dst.cpu().numpy(), want), plan.describe()
