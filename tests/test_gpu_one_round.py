"""GPU parity of the products whose tiles all run at once (gemm_split_sm100.cu), through the C ABI against
the CPU oracle: one row and one column block and their remainders, K in one piece and divided over
clusters of two, four and eight, K of an odd number of stages, a result no 16-byte store can write,
every term of the epilogue, and the weight's NaN codes. Each shape's cut (tile width, CTAs of a cluster)
stands beside it and is asserted, and that it has none into tiles of 256 rows, so that a change of a
rule cannot empty the test. Half rows that the few-row kernels take are left out; bfloat16 ones are in where a
rule sends them here."""
import ctypes

import numpy as np
import pytest

from helpers import check_parity, random_codes, randn

pytestmark = pytest.mark.gpu


def dev(F, arr, dtype):
    return F.Tensor.from_numpy(arr, dtype, F.Device.CUDA)


def matmul(F, a, codes, scale, is_bf16, addend=None):
    dt = F.DType.BFLOAT16 if is_bf16 else F.DType.FLOAT16
    args = dev(F, a, dt), dev(F, codes, F.DType.FP8E4M3), dev(F, np.array([scale], np.float32), F.DType.FLOAT)
    out = F.fp8_matmul(*args) if addend is None else F.fp8_matmul_add(*args, dev(F, addend, dt), expand=True)
    y = out.numpy()
    F.synchronize()
    return y


def cut(F, kind, m, n, k):
    """(tile width, CTAs of a cluster) of a product of half (0), bfloat16 (1) or quantised (2) rows on this card, in
    tiles of 128 rows, which have to be the ones it runs on."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    out = (ctypes.c_int32 * 8)()
    if kind < 2:
        F.check(F.lib().fl_sm100_one_round_pairs(kind, m, n, k, sms, out))
        assert out[0] == 0, "goes to tiles of 256 rows"
    F.check(F.lib().fl_sm100_one_round_plan(kind, m, n, k, sms, 1, out))
    return out[0], out[1]


CUTS = {(77, 2560, 2048): (128, 4), (65, 1288, 640): (32, 2), (127, 136, 272): (32, 2), (128, 1280, 656): (32, 2), (129, 1304, 1040): (64, 2),
        (300, 1280, 640): (64, 2), (131, 9528, 288): (144, 1), (1000, 1280, 1280): (160, 2), (70, 264, 4096): (128, 8), (130, 72, 12288): (128, 8)}
SHAPES = [(77, 2560, 2048), (65, 1288, 640), (127, 136, 272), (128, 1280, 656), (129, 1304, 1040), (300, 1280, 640),
          (131, 9528, 288), (1000, 1280, 1280), (70, 264, 4096), (130, 72, 12288)]


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("is_bf16", [False, True])
@pytest.mark.parametrize("addend", ["none", "bias", "residual"])
def test_matmul(flint, oracle, m, n, k, is_bf16, addend):
    assert cut(flint, int(is_bf16), m, n, k) == CUTS[m, n, k]
    rng = np.random.default_rng(m * 7 + n + k)
    a = oracle.narrow(randn(rng, (m, k)), is_bf16)
    codes = random_codes(rng, n, k)
    add = None if addend == "none" else oracle.narrow(randn(rng, (n,) if addend == "bias" else (m, n)), is_bf16)
    got = matmul(flint, a, codes, 0.0137, is_bf16, add)
    check_parity(oracle, got, oracle.fp8_matmul(a, codes, [np.float32(0.0137)], add, is_bf16), is_bf16, what=f"{m}x{n}x{k}")


@pytest.mark.parametrize("m,n,k,width,split", [(129, 11880, 272, 176, 1), (257, 8712, 272, 192, 1), (65, 11880, 1616, 192, 2),
                                               (129, 2376, 2064, 192, 4), (257, 10296, 272, 224, 1), (129, 7128, 1616, 224, 2),
                                               (257, 11880, 272, 256, 1), (269, 6056, 1488, 256, 2)])
@pytest.mark.parametrize("is_bf16", [False, True])
def test_matmul_in_wide_tiles(flint, oracle, m, n, k, width, split, is_bf16):
    assert cut(flint, int(is_bf16), m, n, k) == (width, split)
    rng = np.random.default_rng(m * 7 + n + k)
    a, codes, add = oracle.narrow(randn(rng, (m, k)), is_bf16), random_codes(rng, n, k), oracle.narrow(randn(rng, (m, n)), is_bf16)
    got = matmul(flint, a, codes, 0.0137, is_bf16, add)
    check_parity(oracle, got, oracle.fp8_matmul(a, codes, [np.float32(0.0137)], add, is_bf16), is_bf16, what=f"{m}x{n}x{k}")


@pytest.mark.parametrize("m,n,k,width,split", [(12, 12288, 2048, 192, 2), (16, 16384, 3072, 224, 2), (17, 1288, 1040, 32, 2), (32, 3072, 3072, 128, 4),
                                               (64, 2560, 656, 64, 2)])
@pytest.mark.parametrize("addend", ["none", "bias", "residual"])
def test_few_bfloat16_rows(flint, oracle, m, n, k, width, split, addend):
    """Twelve to sixteen rows against many channels, and up to 64, which only half rows have a kernel for."""
    assert cut(flint, 1, m, n, k) == (width, split)
    rng = np.random.default_rng(m * 7 + n + k)
    a, codes = oracle.narrow(randn(rng, (m, k)), True), random_codes(rng, n, k)
    add = None if addend == "none" else oracle.narrow(randn(rng, (n,) if addend == "bias" else (m, n)), True)
    before = flint.launch_count()
    got = matmul(flint, a, codes, 0.0137, True, add)
    assert flint.launch_count() == before + 1  # no pass that widens the weight
    check_parity(oracle, got, oracle.fp8_matmul(a, codes, [np.float32(0.0137)], add, True), True, what=f"{m}x{n}x{k}")


@pytest.mark.parametrize("is_bf16", [False, True])
def test_a_residual_that_repeats(flint, oracle, is_bf16):
    """An addend of 67 rows under three blocks of 67: it repeats with a period that is no tile's."""
    F = flint
    dt = F.DType.BFLOAT16 if is_bf16 else F.DType.FLOAT16
    rng = np.random.default_rng(8)
    n, k = 1288, 1040
    assert cut(F, int(is_bf16), 3 * 67, n, k) == (64, 2)
    a, codes, add = oracle.narrow(randn(rng, (3, 67, k)), is_bf16), random_codes(rng, n, k), oracle.narrow(randn(rng, (67, n)), is_bf16)
    out = F.Tensor.empty((3, 67, n), dt)
    args = dev(F, a, dt), dev(F, codes, F.DType.FP8E4M3), dev(F, np.array([0.0137], np.float32), F.DType.FLOAT), dev(F, add, dt), out
    before = F.launch_count()
    F.check(F.lib().fl_fp8_matmul_add(*(t.raw() for t in args)))
    assert F.launch_count() == before + 1  # nothing was expanded
    got = out.numpy().reshape(3 * 67, n)
    F.synchronize()
    want = oracle.fp8_matmul(a.reshape(3 * 67, k), codes, [np.float32(0.0137)], np.tile(add, (3, 1)), is_bf16)
    check_parity(oracle, got, want, is_bf16, what="periodic residual")


LINEAR_CUTS = {(65, 1288, 656): (32, 1), (128, 3072, 3072): (32, 1), (200, 640, 2064): (32, 1), (257, 1280, 256): (32, 1), (700, 640, 272): (32, 1),
               (1024, 1280, 1280): (80, 1), (90, 72, 12288): (0, 0),  # (the persistent kernel, K in halves)
               (33, 4840, 256): (48, 1), (33, 7128, 272): (64, 1), (33, 11880, 256): (96, 1), (129, 7128, 256): (112, 1), (129, 10824, 272): (160, 1),
               (129, 13112, 256): (192, 1), (257, 10296, 256): (224, 1), (257, 11880, 1040): (256, 1)}


@pytest.mark.parametrize("m,n,k", [(33, 4840, 256), (33, 7128, 272), (33, 11880, 256), (129, 7128, 256), (129, 10824, 272), (129, 13112, 256),
                                   (257, 10296, 256), (257, 11880, 1040)])
def test_linear_in_tiles_of_every_width(flint, oracle, m, n, k):
    test_linear_with_every_term(flint, oracle, m, n, k, True)


@pytest.mark.parametrize("m,n,k", [(65, 1288, 656), (128, 3072, 3072), (200, 640, 2064), (257, 1280, 256), (700, 640, 272),
                                   (1024, 1280, 1280), (90, 72, 12288)])
@pytest.mark.parametrize("is_bf16", [True, False])
def test_linear_with_every_term(flint, oracle, m, n, k, is_bf16):
    F = flint
    assert cut(F, 2, m, n, k) == LINEAR_CUTS[m, n, k]
    rng = np.random.default_rng(m + n + k)
    dt = F.DType.BFLOAT16 if is_bf16 else F.DType.FLOAT16
    x = oracle.narrow(randn(rng, (m, k)), is_bf16)
    codes, scales = oracle.quantize_fp8_rows(randn(rng, (n, k), 0.02))
    bias, res = oracle.narrow(randn(rng, (n,), 0.1), is_bf16), oracle.narrow(randn(rng, (m, n)), is_bf16)
    got = F.fp8_linear(dev(F, x, dt), dev(F, codes, F.DType.FP8E4M3), dev(F, scales, F.DType.FLOAT), dev(F, bias, dt),
                       dev(F, res, dt), F.ACT_GELU_TANH).numpy()
    F.synchronize()
    check_parity(oracle, got, oracle.fp8_linear(x, codes, scales, bias, res, oracle.ACT_GELU_TANH, is_bf16), is_bf16,
                 what=f"{m}x{n}x{k}")


def test_results_off_a_16_byte_boundary(flint, oracle):
    F = flint
    rng = np.random.default_rng(5)
    m, n, k = 100, 264, 512
    assert cut(F, 0, m, n, k)[1] > 0
    a, codes = oracle.narrow(randn(rng, (m, k)), False), random_codes(rng, n, k)
    store = F.Tensor.from_numpy(np.zeros(m * n + 8, np.uint16), F.DType.FLOAT16, F.Device.CUDA)
    out = store.view_as((m, n), (n, 1), 1)
    ta, tw, ts = dev(F, a, F.DType.FLOAT16), dev(F, codes, F.DType.FP8E4M3), dev(F, np.array([0.01], np.float32), F.DType.FLOAT)
    F.check(F.lib().fl_fp8_matmul(ta.raw(), tw.raw(), ts.raw(), out.raw()))
    got = store.numpy()
    F.synchronize()
    assert got[0] == 0 and not got[m * n + 1:].any()
    check_parity(oracle, got[1:m * n + 1].reshape(m, n), oracle.fp8_matmul(a, codes, [np.float32(0.01)]), False, what="offset result")


@pytest.mark.parametrize("is_bf16", [False, True])
def test_nan_codes_stay_nan(flint, oracle, is_bf16):
    rng = np.random.default_rng(6)
    m, n, k = 80, 1280, 640
    assert cut(flint, int(is_bf16), m, n, k)[1] > 0
    a, codes = oracle.narrow(randn(rng, (m, k)), is_bf16), random_codes(rng, n, k)
    codes[3, 17], codes[700, 639] = 0x7F, 0xFF
    y = oracle.widen(matmul(flint, a, codes, 0.0137, is_bf16), is_bf16)
    assert np.isnan(y[:, [3, 700]]).all()
    assert np.isfinite(np.delete(y, [3, 700], axis=1)).all()


@pytest.mark.parametrize("m,k", [(592, 16), (593, 1040), (601, 2064), (600, 3072), (700, 3088), (592, 4096)])
@pytest.mark.parametrize("is_bf16", [True, False])
def test_a_warp_to_a_row_quantises_bit_exactly(flint, oracle, m, k, is_bf16):
    """Either side of quantize_fp8_act_warp_kernel's range in k (its rows are below)."""
    F = flint
    rng = np.random.default_rng(m + k)
    x = randn(rng, (m, k))
    x[1] = 0
    x[2, k - 1], x[3, 0] = 90.0, -3e4
    x[4] *= 1e-6
    x16 = oracle.narrow(x, is_bf16)
    t = dev(F, x16, F.DType.BFLOAT16 if is_bf16 else F.DType.FLOAT16)
    codes, scales = F.Tensor.empty((m, k), F.DType.FP8E4M3), F.Tensor.empty((m,), F.DType.FLOAT)
    F.check(F.lib().fl_quantize_fp8_activation(t.raw(), codes.raw(), scales.raw()))
    want_codes, want_scales = oracle.quantize_fp8_act(x16, is_bf16)
    assert np.array_equal(scales.numpy().view(np.uint32), want_scales.view(np.uint32))
    assert np.array_equal(codes.numpy(), want_codes)


@pytest.mark.parametrize("m,k", [(592, 16), (593, 768), (592, 784), (1480, 784), (1481, 1024), (1487, 1040), (1480, 2048), (1480, 2064),
                                 (3551, 2064), (3552, 2064), (3555, 3072), (3552, 3088)])
@pytest.mark.parametrize("is_bf16", [True, False])
def test_rows_with_nans_and_infinities_quantise_bit_exactly(flint, oracle, m, k, is_bf16):
    """quantize_fp8_act_warp_kernel (rows of up to 768 from 592 of them on, of up to 2048 from 1480, of
    up to 3072 from 3552) and
    its neighbours: a row's maximum passes over its NaNs, whichever half of a pair they are in, an
    infinity makes the scale one, and a row of NaNs has scale 0."""
    F = flint
    rng = np.random.default_rng(m + 3 * k)
    x = randn(rng, (m, k))
    x[0], x[1, :] = 0, np.nan
    x[2, 0], x[3, k - 1], x[4, 1] = np.nan, np.nan, -np.nan
    x[5, 3], x[6, k - 2], x[7, 0], x[7, 1] = np.inf, -np.inf, np.nan, np.inf
    x[m - 1, k - 1], x[m - 2] = 3e4, 1e-7 * x[m - 2]
    x16 = oracle.narrow(x, is_bf16)
    t = dev(F, x16, F.DType.BFLOAT16 if is_bf16 else F.DType.FLOAT16)
    codes, scales = F.Tensor.empty((m, k), F.DType.FP8E4M3), F.Tensor.empty((m,), F.DType.FLOAT)
    F.check(F.lib().fl_quantize_fp8_activation(t.raw(), codes.raw(), scales.raw()))
    want_codes, want_scales = oracle.quantize_fp8_act(x16, is_bf16)
    assert np.array_equal(scales.numpy().view(np.uint32), want_scales.view(np.uint32))
    assert np.array_equal(codes.numpy(), want_codes)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("n,h,hk,L,S", [(2, 3, 3, 600, 600), (1, 4, 2, 260, 900), (3, 2, 1, 385, 385)])
def test_causal_units_of_several_heads(flint, oracle, n, h, hk, L, S, d):
    """The order of the causal masks' units over heads and batches, a last unit with one tile of
    queries, and a first tile that stops before the second."""
    F = flint
    rng = np.random.default_rng(L + S + d)
    q, k, v = (oracle.narrow(randn(rng, s), True) for s in ((n, h, L, d), (n, hk, S, d), (n, hk, S, d)))
    out = F.attention(*(dev(F, t, F.DType.BFLOAT16) for t in (q, k, v)), 1, 0)
    got = oracle.widen(out.numpy(), True).astype(np.float64)
    F.synchronize()
    want = oracle.attention(q, k, v, True, True)
    assert oracle.rel_l2(got, want) <= 5e-3
    assert np.abs(got - want).max() <= 2 * oracle.ulp16_at(float(np.abs(want).max()), True)


@pytest.mark.parametrize("block_size", [64, 100, 128, 257, 400])
@pytest.mark.parametrize("n,h,hk,L,S,d", [(2, 3, 3, 600, 600, 64), (1, 4, 2, 260, 900, 128), (3, 2, 1, 385, 385, 128)])
def test_block_causal_units_of_several_heads(flint, oracle, n, h, hk, L, S, d, block_size):
    """The same under the block-causal mask: blocks below a tile of keys, across its boundary, of a tile and
    wider than two, so that both tiles of a unit may end on the same block of keys or on different ones."""
    F = flint
    rng = np.random.default_rng(L + S + d + block_size)
    q, k, v = (oracle.narrow(randn(rng, s), True) for s in ((n, h, L, d), (n, hk, S, d), (n, hk, S, d)))
    out = F.attention(*(dev(F, t, F.DType.BFLOAT16) for t in (q, k, v)), 2, block_size)
    got = oracle.widen(out.numpy(), True).astype(np.float64)
    F.synchronize()
    want = oracle.attention(q, k, v, 2, True, block_size)
    assert oracle.rel_l2(got, want) <= 5e-3
    assert np.abs(got - want).max() <= 2 * oracle.ulp16_at(float(np.abs(want).max()), True)


@pytest.mark.parametrize("m,n,k", [(260, 9488, 5376), (814, 4816, 11120), (1024, 384, 12288), (300, 1280, 1280), (200, 2584, 880),
                                   (128, 3072, 3072)])
def test_linears_on_quantised_rows_give_the_same_bits(flint, m, n, k):
    """fl_fp8_linear, which takes the one-round kernel where that is faster, against the forms that run on
    the persistent kernel alone (row maxima, several destinations): where that kernel cuts a tile's
    K in two, as in the first three shapes, and where it does not, the sums are the same."""
    import torch
    F = flint
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    bf = F.DType.BFLOAT16

    def new(shape, std, kind=torch.bfloat16, dtype=bf):
        t = (torch.randn(shape, device="cuda", generator=gen) * std).to(kind)
        return F.Tensor.from_device_ptr(t.data_ptr(), shape, dtype, keepalive=t)

    x, bias, res = new((m, k), 1.0), new((n,), 0.1), new((m, n), 1.0)
    codes, scales = F.quantize_fp8_rows(new((n, k), 0.02, torch.float32, F.DType.FLOAT))
    want = F.fp8_linear(x, codes, scales, bias, res, F.ACT_GELU_TANH).numpy()
    row_amax = F.Tensor.empty((m,), F.DType.FLOAT)
    got = F.fp8_linear_amax(x, codes, scales, row_amax, bias, res, F.ACT_GELU_TANH).numpy()
    assert np.array_equal(got, want), "with the rows' maxima"
    wide = F.Tensor.empty((m, n + 8), bf)
    F.fp8_linear_scatter(x, codes, scales, [wide], 8, bias, res, F.ACT_GELU_TANH)
    assert np.array_equal(wide.numpy()[:, 8:], want), "into a column block"
    xc, xs = F.Tensor.empty((m, k), F.DType.FP8E4M3), F.Tensor.empty((m,), F.DType.FLOAT)
    F.check(F.lib().fl_quantize_fp8_activation(x.raw(), xc.raw(), xs.raw()))
    out = F.Tensor.empty((m, n), bf)
    F.fp8_linear_quantized(xc, xs, codes, scales, bias, res, F.ACT_GELU_TANH, out)
    assert np.array_equal(out.numpy(), want), "on rows quantised beforehand"
    if cut(F, 2, m, n, k)[1] > 0:  # (without its workspace the persistent kernel cuts nothing)
        F.fp8_linear_static(x, codes, scales, bias, res, F.ACT_GELU_TANH, out)
        assert np.array_equal(out.numpy(), want), "without an allocation"
    F.synchronize()
