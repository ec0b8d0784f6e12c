"""GPU parity of the one-round kernel's tiles of 256 rows (fl_fp8_matmul[_add] on more than one row block
against an e4m3 weight) with the oracle: every tile width that the rule takes, row counts that leave a pair's
second CTA few rows or none, columns and K that end inside a tile and a stage. Each shape's width stands beside
it and is asserted. Tolerances as in test_gpu_one_round.py."""
import os
import subprocess
import sys

import numpy as np
import pytest

from helpers import check_parity, random_codes, randn
from test_gpu_one_round import matmul
from test_one_round_pairs_cpu import pairs

pytestmark = pytest.mark.gpu

# m, n, k, and the tile width for half and for bfloat16 rows (0: no tiles of 256 rows, and the case is left out). The
# last five leave the second CTA of the last row block without a row.
CASES = [(396, 3496, 1312, 96, 96), (663, 2832, 1152, 128, 128), (129, 8632, 2704, 128, 128), (512, 5120, 3072, 160, 160),
         (1705, 1400, 3696, 160, 160), (238, 14088, 2304, 192, 192), (385, 7048, 3088, 192, 192), (256, 16384, 3072, 0, 224),
         (399, 9096, 272, 0, 256), (1299, 1528, 1120, 128, 128), (1284, 1888, 944, 160, 160), (1293, 2296, 464, 192, 192),
         (1320, 2304, 288, 0, 192), (778, 4528, 1168, 0, 256)]


def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("m,n,k,width,is_bf16", [(*c[:3], c[3 + is_bf16], bool(is_bf16)) for c in CASES for is_bf16 in (0, 1) if c[3 + is_bf16]])
@pytest.mark.parametrize("addend", ["none", "bias", "residual"])
def test_matmul_in_pairs(flint, oracle, m, n, k, width, is_bf16, addend):
    assert pairs(int(is_bf16), m, n, k, sms())["block_n"] == width
    rng = np.random.default_rng(m + n + k)
    a = oracle.narrow(randn(rng, (m, k)), is_bf16)
    codes = random_codes(rng, n, k)
    add = None if addend == "none" else oracle.narrow(randn(rng, (n,) if addend == "bias" else (m, n)), is_bf16)
    got = matmul(flint, a, codes, 0.0137, is_bf16, add)
    check_parity(oracle, got, oracle.fp8_matmul(a, codes, [np.float32(0.0137)], add, is_bf16), is_bf16, what=f"{m}x{n}x{k}")


@pytest.mark.parametrize("is_bf16", [False, True])
def test_nan_codes_stay_nan_in_pairs(flint, oracle, is_bf16):
    rng = np.random.default_rng(8)
    m, n, k = 663, 2832, 1152
    assert pairs(int(is_bf16), m, n, k, 148)["block_n"] > 0
    a, codes = oracle.narrow(randn(rng, (m, k)), is_bf16), random_codes(rng, n, k)
    codes[3, 17], codes[2700, 1151] = 0x7F, 0xFF
    y = oracle.widen(matmul(flint, a, codes, 0.0137, is_bf16), is_bf16)
    assert np.isnan(y[:, [3, 2700]]).all()
    assert np.isfinite(np.delete(y, [3, 2700], axis=1)).all()


SINGLE = """
import sys
sys.path[:0] = sys.argv[1:3]
import numpy as np
from libwaifu_b200 import flint
from oracle import oracle
from helpers import check_parity, random_codes, randn
from test_gpu_one_round import matmul
from test_one_round_pairs_cpu import pairs
rng = np.random.default_rng(4)
for m, n, k in [(663, 2832, 1152), (1440, 2176, 1504)]:
    for is_bf16 in (True, False):
        assert pairs(int(is_bf16), m, n, k)["block_n"] == 0
        a, codes = oracle.narrow(randn(rng, (m, k)), is_bf16), random_codes(rng, n, k)
        got = matmul(flint, a, codes, 0.0137, is_bf16)
        check_parity(oracle, got, oracle.fp8_matmul(a, codes, [np.float32(0.0137)], None, is_bf16), is_bf16, what=f"{m}x{n}x{k}")
"""


def test_products_that_have_pairs_run_without_them(flint):
    """Under FLINT_SM100_SINGLE_CTA=1, on tiles of 128 rows and, the second shape, on the persistent kernel, for
    which bfloat16 rows want the weight widened beforehand."""
    here = os.path.dirname(os.path.abspath(__file__))
    assert all(pairs(kind, 1440, 2176, 1504)["block_n"] for kind in (0, 1))
    subprocess.run([sys.executable, "-c", SINGLE, here, os.path.dirname(here)], env=dict(os.environ, FLINT_SM100_SINGLE_CTA="1"), check=True,
                   timeout=300)
