"""The DRAM traffic that bench.py reports beside its kernels (CPU): a 512^3 complex128 pass or move reads and writes its
array once, and all that can be missing from the counters is what is still in L2 (129 MB) when the kernel ends."""
import json
import os

import pytest

PATH = os.path.join(os.path.dirname(__file__), "..", "profiles", "traffic.json")
ALGORITHMIC = 2 * 512 ** 3 * 16


@pytest.mark.parametrize("kernel", ["reshape_512c128_block_to_rotate", "fft_pass_512c128", "fft_pass_fp64_512c128"])
def test_traffic_is_the_arrays_read_and_written_once(kernel):
    with open(PATH) as f:
        got = json.load(f)[kernel]
    assert ALGORITHMIC - 129e6 <= got <= 1.05 * ALGORITHMIC
