"""Relative L2 errors of one forward transform per arithmetic and kernel form against longer arithmetic (GPU), with limits
close enough to see a stage that lost a bit or two or a constant whose bias came back (the oracle tests allow some thirty
times the error).

A level of a transform (a factor of two in the length) rounds every value about once, by at most u, and levels add in
quadrature: u sqrt(log2 N), with u = 2^-53 in native FP64, 2^-24 in FP32, and 2^-48 in double-float (two 24-bit parts)."""
import math

import numpy as np
import pytest

from decomp_mpi_gb300 import api
from tests.test_reg_accuracy import LONG, _arrays, _errors

pytestmark = pytest.mark.gpu
ARITH = {"fp64": (api.C128, api.ARITH_FP64, 2.0 ** -53), "fp32": (api.C64, api.ARITH_FP32, 2.0 ** -24),
         "df": (api.C128, api.ARITH_DF, 2.0 ** -48)}


@pytest.mark.skipif(not LONG, reason="no longer float on the host")
@pytest.mark.parametrize("along_t", [False, True], ids=["v1", "t"])
@pytest.mark.parametrize("name", list(ARITH))
@pytest.mark.parametrize("n", [48, 105, 243, 512, 1024])
def test_forward(n, name, along_t, cuda):
    dtype, arith, u = ARITH[name]
    shape, arrays = _arrays(n, along_t)
    err, _ = _errors(cuda, arrays[:64], shape, dtype, arith, [lambda plan: None])
    assert err[0] <= u * math.sqrt(math.log2(float(np.prod(shape)))), err
