"""GPU parity of the products whose tiles all run at once (gemm_split_sm100.cu), through the C ABI against
the CPU oracle: one row and one column block and their remainders, K in one piece and divided over
clusters of two, four and eight, K of an odd number of stages, a result no 16-byte store can write,
every term of the epilogue, and the weight's NaN codes. Sizes that earlier dispatch rules send
elsewhere (few rows) are left out."""
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


SHAPES = [(77, 2560, 2048), (65, 1288, 640), (127, 136, 272), (128, 1280, 656), (129, 1304, 1040), (300, 1280, 640),
          (512, 5120, 784), (1000, 1280, 1280), (70, 264, 4096), (130, 72, 12288)]


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("is_bf16", [False, True])
@pytest.mark.parametrize("addend", ["none", "bias", "residual"])
def test_matmul(flint, oracle, m, n, k, is_bf16, addend):
    rng = np.random.default_rng(m * 7 + n + k)
    a = oracle.narrow(randn(rng, (m, k)), is_bf16)
    codes = random_codes(rng, n, k)
    add = None if addend == "none" else oracle.narrow(randn(rng, (n,) if addend == "bias" else (m, n)), is_bf16)
    got = matmul(flint, a, codes, 0.0137, is_bf16, add)
    check_parity(oracle, got, oracle.fp8_matmul(a, codes, [np.float32(0.0137)], add, is_bf16), is_bf16, what=f"{m}x{n}x{k}")


@pytest.mark.parametrize("m,n,k", [(65, 1288, 656), (128, 3072, 3072), (200, 640, 2064), (257, 1280, 256), (700, 640, 272),
                                   (1024, 1280, 1280), (90, 72, 12288)])
@pytest.mark.parametrize("is_bf16", [True, False])
def test_linear_with_every_term(flint, oracle, m, n, k, is_bf16):
    F = flint
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


@pytest.mark.parametrize("m,k", [(592, 16), (593, 768), (592, 784), (1480, 784), (1481, 1024), (1487, 1040), (1480, 2048), (1480, 2064)])
@pytest.mark.parametrize("is_bf16", [True, False])
def test_rows_with_nans_and_infinities_quantise_bit_exactly(flint, oracle, m, k, is_bf16):
    """quantize_fp8_act_warp_kernel (rows of up to 768 from 592 of them on, of up to 2048 from 1480) and
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
    F.synchronize()
