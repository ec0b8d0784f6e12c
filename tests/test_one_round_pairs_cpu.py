"""The one-round kernel's tiles of 256 rows (a pair of CTAs each), their index arithmetic without a GPU."""
import ctypes
import os
import random
import subprocess
import sys

import pytest

from libwaifu_b200 import flint as F

NAMES = ("block_n", "split", "ctas", "num_kb", "load_slots", "wide_slots", "slot_bytes", "smem")


def pairs(kind, m, n, k, sms=148):
    out = (ctypes.c_int32 * 8)()
    F.check(F.lib().fl_sm100_one_round_pairs(kind, m, n, k, sms, out))
    return dict(zip(NAMES, out))


@pytest.mark.parametrize("sms", [148, 132, 16, 2])
@pytest.mark.parametrize("kind", [0, 1])
def test_pair_invariants(kind, sms):
    """All pairs are resident at once; a CTA's half of the columns is whole 16-row groups whose slots stay
    on 1024-byte boundaries; rings and exchange buffer fit; a ring of loads holds whole turns of the
    widened ring, so that a warp meets every phase of its barriers."""
    rng = random.Random(23)
    taken = 0
    for _ in range(3000):
        m, n, k = int(2 ** rng.uniform(0, 13)), 8 * int(2 ** rng.uniform(0, 11.2)), 16 * int(2 ** rng.uniform(0, 9.7))
        p = pairs(kind, m, n, k, sms)
        if p["block_n"] == 0:
            assert not any(p.values())
            continue
        taken += 1
        what = f"{m}x{n}x{k} {p}"
        half = p["block_n"] // 2
        assert m > 128 and p["split"] == 1 and 64 <= p["block_n"] <= 256 and p["block_n"] % 32 == 0, what
        assert p["num_kb"] == -(-k * 2 // 128)
        assert p["ctas"] == -(-m // 256) * -(-n // p["block_n"]) * 2 and p["ctas"] <= sms, what
        assert p["slot_bytes"] == 128 * 128 + half * 64 and p["slot_bytes"] % 1024 == 0 and half * 128 % 1024 == 0, what
        assert p["wide_slots"] in (2, 4) and 1 <= p["load_slots"] <= 8 and p["load_slots"] % p["wide_slots"] == 0, what
        assert p["smem"] - 1024 >= p["load_slots"] * p["slot_bytes"] + p["wide_slots"] * half * 128, what
        assert p["smem"] - 1024 >= p["block_n"] // 4 * (128 * 16 + 16) and p["smem"] <= 227 * 1024 - 1024, what
    assert taken > 0 or sms < 132


def test_refusals():
    out = (ctypes.c_int32 * 8)()
    for bad in [(2, 200, 8, 16, 148), (-1, 200, 8, 16, 148), (0, 0, 8, 16, 148), (0, 200, 8, 16, 1)]:
        assert F.lib().fl_sm100_one_round_pairs(*bad, out) == F.FL_ERROR_INVALID_ARG
    assert F.lib().fl_sm100_one_round_pairs(0, 200, 8, 16, 148, None) == F.FL_ERROR_INVALID_ARG


def test_no_pairs_where_single_ctas_were_asked_for():
    """FLINT_SM100_SINGLE_CTA=1, read when a process first asks: no tile of 256 rows, which pairs CTAs."""
    script = ("import sys; sys.path[:0] = [%r, %r]; from test_one_round_pairs_cpu import pairs; "
              "print([pairs(kind, 512, 5120, 3072)['block_n'] for kind in (0, 1)])"
              % (os.path.dirname(os.path.abspath(__file__)), os.path.dirname(os.path.dirname(os.path.abspath(__file__)))))
    said = [subprocess.run([sys.executable, "-c", script], env=dict(os.environ, FLINT_SM100_SINGLE_CTA=flag), check=True, capture_output=True,
                           text=True).stdout.strip() for flag in ("1", "0")]
    assert said == ["[0, 0]", "[160, 160]"]


def test_half_rows_of_a_short_k_that_measured_slower_in_pairs():
    """Either side of the second line, and bfloat16 rows of the same shapes, whose other ways take longer."""
    for m, n, k in [(1593, 1696, 816), (1553, 1856, 672), (569, 4528, 1088), (1031, 2488, 1008), (423, 4936, 880), (1978, 1296, 1088)]:
        assert pairs(0, m, n, k)["block_n"] == 0, (m, n, k)
        assert pairs(1, m, n, k)["block_n"] > 128, (m, n, k)
    for m, n, k in [(486, 4424, 1072), (234, 8840, 1136), (904, 2080, 1296), (2001, 1632, 1120), (689, 4472, 1008), (1940, 1648, 1344)]:
        assert pairs(0, m, n, k)["block_n"] > 0, (m, n, k)
