"""Which form of the two-tile attention kernel a call takes, as host arithmetic: the line between them at shapes that
were measured on both sides of it."""
import pytest

from libwaifu_b200 import flint as F

NONE, CAUSAL, BLOCK_CAUSAL, BLOCK_DIAGONAL = range(4)


def takes_over(batch, heads, q_len, kv_len, head_dim, mask, block=0, sms=148):
    return F.lib().fl_sm100_attention_takes_over(batch, heads, q_len, kv_len, head_dim, mask, block, sms)


@pytest.mark.parametrize("shape", [
    (1, 24, 2048, 2048, 128, CAUSAL), (1, 18, 2048, 2048, 128, CAUSAL), (1, 27, 1792, 1792, 128, CAUSAL), (1, 20, 1536, 1536, 128, CAUSAL),
    (1, 24, 1024, 1024, 128, NONE), (1, 37, 1024, 1024, 128, NONE), (1, 27, 768, 768, 128, NONE), (1, 100, 129, 1024, 128, NONE),
    (1, 24, 1200, 2000, 128, BLOCK_CAUSAL, 1900), (1, 17, 1536, 1536, 128, BLOCK_CAUSAL, 1382), (1, 12, 2048, 2048, 128, BLOCK_CAUSAL, 921),
    (2, 24, 4352, 4352, 128, NONE), (1, 24, 2048, 2048, 128, NONE), (1, 160, 140, 2049, 64, CAUSAL), (1, 24, 1024, 1025, 64, NONE)])
def test_the_longest_chain_keeps_the_kernel_of_one_unit(shape):
    assert takes_over(*shape) == 0


@pytest.mark.parametrize("shape", [
    (4, 32, 1000, 1000, 128, CAUSAL), (1, 28, 2048, 2048, 128, CAUSAL), (1, 50, 1536, 1536, 128, CAUSAL), (1, 100, 256, 256, 128, CAUSAL),
    (1, 10, 1536, 1536, 128, CAUSAL), (1, 6, 2048, 2048, 128, CAUSAL), (3, 24, 1000, 1000, 128, NONE), (1, 42, 1024, 1024, 128, NONE),
    (1, 12, 1024, 1024, 128, NONE), (1, 74, 512, 512, 128, NONE), (2, 24, 2048, 2048, 128, BLOCK_CAUSAL, 1024), (4, 32, 1000, 1000, 128, BLOCK_CAUSAL, 64),
    (1, 24, 2048, 2048, 64, CAUSAL), (1, 24, 1024, 1024, 64, NONE), (1, 24, 1200, 2000, 64, BLOCK_CAUSAL, 1900), (2, 8, 300, 300, 128, BLOCK_DIAGONAL, 300)])
def test_short_walks_and_full_gpus_go_on(shape):
    assert takes_over(*shape) == 1


def test_calls_of_one_tile_have_nothing_to_take_over():
    assert takes_over(1, 500, 128, 256, 64, NONE) == 0 and takes_over(2, 90, 300, 300, 64, BLOCK_DIAGONAL, 48) == 0


def test_refusals():
    for bad in [(0, 1, 200, 200, 64, NONE), (1, 1, 200, 200, 96, NONE), (1, 1, 200, 100, 64, CAUSAL), (1, 1, 200, 200, 64, BLOCK_CAUSAL, 0)]:
        assert takes_over(*bad) == -1
    assert takes_over(1, 1, 200, 200, 64, NONE, 0, 0) == -1
