"""The one-round kernel's cut of a product, checked without a GPU: what its index arithmetic relies on.
Every K stage of a tile belongs to one rank of its cluster; the column blocks that the ranks finish are
whole 16-column chunks; all CTAs are resident at once; rings and exchange buffer fit the shared memory; a
ring of loads holds whole turns of the widened ring, so that a warp meets every phase of its barriers;
and quantised rows, whose results are the persistent kernel's bits, are neither divided nor taken where
that kernel cuts a tile's K."""
import ctypes
import random

import pytest

from libwaifu_b200 import flint as F
from test_gemm_schedule_cpu import plan as tile_plan

HALF, BF16, QUANTISED = 0, 1, 2
NAMES = ("block_n", "split", "ctas", "num_kb", "load_slots", "wide_slots", "slot_bytes", "smem")


def plan(kind, m, n, k, sms=148, allow=1):
    out = (ctypes.c_int32 * 8)()
    F.check(F.lib().fl_sm100_one_round_plan(kind, m, n, k, sms, allow, out))
    return dict(zip(NAMES, out))


def shapes():
    rng = random.Random(17)
    yield from [(77, 2560, 2048), (512, 5120, 3072), (1, 8, 16), (128, 16, 64), (129, 1304, 1040), (4096, 136, 12288), (16, 16384, 4096)]
    for _ in range(1500):
        yield (int(2 ** rng.uniform(0, 13)), 8 * int(2 ** rng.uniform(0, 11.2)), 16 * int(2 ** rng.uniform(0, 9.7)))


@pytest.mark.parametrize("sms", [148, 132, 16, 2])
@pytest.mark.parametrize("kind", [HALF, BF16, QUANTISED])
def test_plan_invariants(kind, sms):
    taken = 0
    for m, n, k in shapes():
        for allow in (0, 1):
            p = plan(kind, m, n, k, sms, allow)
            if p["block_n"] == 0:
                assert not any(p.values())
                continue
            taken += 1
            what = f"{m}x{n}x{k} {p}"
            block_n, split, num_kb = p["block_n"], p["split"], p["num_kb"]
            assert num_kb == -(-k * (1 if kind == QUANTISED else 2) // 128)
            assert 32 <= block_n <= 256 and split in (1, 2, 4, 8) and block_n % (16 * split) == 0, what
            assert p["ctas"] == -(-m // 128) * -(-n // block_n) * split and p["ctas"] <= sms, what
            ranks = [(num_kb * r // split, num_kb * (r + 1) // split) for r in range(split)]
            assert ranks[0][0] == 0 and ranks[-1][1] == num_kb
            assert all(a < b for a, b in ranks) and all(x[1] == y[0] for x, y in zip(ranks, ranks[1:])), what
            assert p["slot_bytes"] == 128 * 128 + block_n * (128 if kind == QUANTISED else 64) and p["slot_bytes"] % 1024 == 0
            assert 1 <= p["load_slots"] <= 8, what
            wide = 0
            if kind == QUANTISED:
                assert split == 1 and p["wide_slots"] == 0, what
                assert not allow or tile_plan("e4m3", m, n, k, sms)["sk_tiles"] == 0, what
            else:
                assert p["wide_slots"] in (2, 4) and p["load_slots"] % p["wide_slots"] == 0, what
                wide = p["wide_slots"] * block_n * 128
            # what is added to the rings is the way up to a 1024-byte boundary
            assert p["smem"] - 1024 >= p["load_slots"] * p["slot_bytes"] + wide, what
            assert p["smem"] - 1024 >= block_n // 4 * (128 * 16 + 16), what
            assert p["smem"] <= 227 * 1024 - 1024, what
    assert taken > 0 or sms == 2


def test_widths_and_clusters_of_the_measured_shapes():
    cut = lambda *a: (plan(*a)["block_n"], plan(*a)["split"])
    assert cut(HALF, 77, 2560, 2048) == (128, 4) and cut(BF16, 512, 5120, 3072) == (160, 1)
    assert cut(QUANTISED, 300, 1280, 1280) == (32, 1) and cut(QUANTISED, 128, 3072, 3072) == (32, 1)
    assert cut(HALF, 4096, 12288, 3072) == (0, 0) and cut(QUANTISED, 4352, 12288, 3072) == (0, 0)
    # the persistent kernel cuts these in two; with no workspace it would not
    assert cut(QUANTISED, 260, 9488, 5376) == (0, 0) and plan(QUANTISED, 260, 9488, 5376, 148, 0)["split"] == 1


def test_products_that_measured_slower_stay_with_the_persistent_kernel():
    """The line between the two kernels at shapes measured on both sides of it."""
    for m, n, k in [(1547, 2024, 2912), (1578, 2080, 1936), (1211, 2144, 9488), (1190, 2256, 11008), (1687, 1536, 9600),
                    (1024, 3072, 12288)]:
        assert plan(BF16, m, n, k)["split"] == 0, (m, n, k)
    for m, n, k in [(938, 2256, 6512), (1342, 1672, 7120), (271, 6888, 7728), (244, 9968, 8272)]:
        assert plan(QUANTISED, m, n, k)["split"] == 0, (m, n, k)
    for kind, m, n, k in [(HALF, 216, 11544, 1280), (HALF, 286, 12000, 1008), (BF16, 868, 5208, 2256), (BF16, 100, 1280, 32768),
                          (BF16, 367, 8792, 11296),
                          (QUANTISED, 1342, 1672, 7104), (QUANTISED, 297, 11472, 2704), (QUANTISED, 36, 880, 9552)]:
        assert plan(kind, m, n, k)["split"] > 0, (m, n, k)


def test_refusals():
    out = (ctypes.c_int32 * 8)()
    for bad in [(3, 1, 8, 16, 148), (-1, 1, 8, 16, 148), (0, 0, 8, 16, 148), (0, 1, 8, 16, 1)]:
        assert F.lib().fl_sm100_one_round_plan(*bad, 1, out) == F.FL_ERROR_INVALID_ARG
    assert F.lib().fl_sm100_one_round_plan(0, 1, 8, 16, 148, 1, None) == F.FL_ERROR_INVALID_ARG


def test_bfloat16_rows_that_no_few_row_kernel_takes():
    route = F.lib().fl_sm100_few_rows_route
    route.argtypes, route.restype = [ctypes.c_int32] * 4, ctypes.c_int32
    MMA_SYNC, NONE = 1, 0
    for m, n, k in [(12, 12288, 2048), (16, 16384, 3072), (17, 3072, 3072), (32, 3072, 3072)]:
        assert route(4, m, n, k) == NONE and plan(BF16, m, n, k)["split"] > 0
    for m, n, k in [(1, 16384, 3072), (11, 16384, 3072), (16, 12280, 3072), (16, 16384, 2032)]:
        assert route(4, m, n, k) == MMA_SYNC
