"""Parity of the one-pass LayerNorm and RMSNorm-layer kernels against the op-by-op restatement of
the reference (layernorm.cu:291-384, RMSNormLayer.cs:156-231), through the function ids a C# layer
would call and through the raw entry points."""
import numpy as np
import pytest

import oracle
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    from mycaffe_b200 import CudaDnn
    c = CudaDnn(0)
    yield c
    c.Dispose()


# (outer, channels, inner): GPT-2 block input, llama width, TFT width, ragged and unaligned rows
SHAPES = [(8, 128, 768), (2, 33, 4096), (4, 192, 64), (3, 7, 1000), (2, 5, 250), (1, 3, 8192), (2, 3, 1539), (1, 2, 16384)]


@pytest.mark.parametrize("outer,channels,inner", SHAPES)
def test_layernorm_ids_match_reference_math(cuda, outer, channels, inner):
    """CREATE_LAYERNORM / LAYERNORM_FWD / LAYERNORM_BWD (ids 970, 975, 976) with the reference's packing."""
    rng = np.random.default_rng(inner)
    x = (rng.standard_normal((outer, channels, inner)) * 1.5 + 0.3).astype(np.float32)
    dy = rng.standard_normal(x.shape).astype(np.float32)
    eps = 1e-5
    h = cuda.CreateLayerNorm(0, x.size, outer, channels, inner, eps)
    hX, hY, hdY, hdX = cuda.AllocMemory(x), cuda.AllocMemory(x.size), cuda.AllocMemory(dy), cuda.AllocMemory(x.size)
    cuda.LayerNormForward(h, hX, hY)
    y = cuda.GetMemory(hY, x.size).reshape(x.shape)
    y_ref, sd = oracle.layernorm_forward(x, eps)
    assert rel_err(y, y_ref) < 1e-5
    cuda.LayerNormBackward(h, hY, hdY, hdX)
    dx = cuda.GetMemory(hdX, x.size).reshape(x.shape)
    dx_ref = oracle.layernorm_backward(y_ref, dy, sd, eps)
    assert rel_err(dx, dx_ref) < 1e-5
    for m in (hX, hY, hdY, hdX):
        cuda.FreeMemory(m)
    cuda.FreeLayerNorm(h)


def test_layernorm_handle_errors(cuda):
    from mycaffe_b200 import CudaDnnError, function_ids as ids
    with pytest.raises(CudaDnnError) as e:
        cuda.CreateLayerNorm(0, 100, 2, 5, 11, 1e-5)   # count != outer * channels * inner
    assert e.value.code == ids.ERROR_PARAM_OUT_OF_RANGE
    with pytest.raises(CudaDnnError) as e:
        cuda.LayerNormForward(12345, 1, 1)
    assert e.value.code == ids.ERROR_LAYERNORM_NOT_INITIALIZED
    h = cuda.CreateLayerNorm(0, 64, 1, 2, 32, 1e-5)
    hA = cuda.AllocMemory(64)
    with pytest.raises(CudaDnnError) as e:
        cuda.LayerNormBackward(h, hA, hA, hA)           # no forward yet: no stdev to divide by
    assert e.value.code == ids.ERROR_LAYERNORM_NOT_INITIALIZED
    cuda.FreeMemory(hA)
    cuda.FreeLayerNorm(h)


@pytest.mark.parametrize("weights", [True, False])
@pytest.mark.parametrize("outer,channels,inner", SHAPES)
def test_rmsnorm_layer_ids_match_reference_math(cuda, outer, channels, inner, weights):
    rng = np.random.default_rng(inner + 1)
    x = rng.standard_normal((outer, channels, inner)).astype(np.float32)
    w = (1 + 0.2 * rng.standard_normal(inner)).astype(np.float32) if weights else None
    dy = rng.standard_normal(x.shape).astype(np.float32)
    eps, rows = 1e-5, outer * channels
    hX, hY, hdY, hdX = cuda.AllocMemory(x), cuda.AllocMemory(x.size), cuda.AllocMemory(dy), cuda.AllocMemory(x.size)
    hInv = cuda.AllocMemory(rows)
    hW = cuda.AllocMemory(w) if weights else 0
    hdW = cuda.AllocMemory(inner) if weights else 0
    cuda.RmsNormForward(hX, hW, hY, hInv, rows, inner, eps)
    y = cuda.GetMemory(hY, x.size).reshape(x.shape)
    y_ref, inv_ref = oracle.rmsnorm_layer_forward(x, w, eps)
    assert rel_err(y, y_ref) < 1e-5
    assert rel_err(cuda.GetMemory(hInv, rows), inv_ref) < 1e-5
    cuda.RmsNormBackward(hX, hW, hdY, hInv, hdX, hdW, rows, inner)
    dx = cuda.GetMemory(hdX, x.size).reshape(x.shape)
    dx_ref, dw_ref = oracle.rmsnorm_layer_backward(x, w, dy, eps)
    assert rel_err(dx, dx_ref) < 1e-5
    if weights:
        assert rel_err(cuda.GetMemory(hdW, inner), dw_ref) < 1e-5
    for m in (hX, hY, hdY, hdX, hInv, hW, hdW):
        if m:
            cuda.FreeMemory(m)


def test_rmsnorm_backward_is_deterministic_and_many_rows(cuda):
    """More rows than CTAs: the weight gradient goes through per-CTA partials added in a fixed order."""
    rng = np.random.default_rng(3)
    rows, inner = 20000, 768
    x = rng.standard_normal((rows, inner)).astype(np.float32)
    w = (1 + 0.1 * rng.standard_normal(inner)).astype(np.float32)
    dy = rng.standard_normal(x.shape).astype(np.float32)
    hX, hW, hdY, hdX = cuda.AllocMemory(x), cuda.AllocMemory(w), cuda.AllocMemory(dy), cuda.AllocMemory(x.size)
    hY, hInv, hdW = cuda.AllocMemory(x.size), cuda.AllocMemory(rows), cuda.AllocMemory(inner)
    cuda.RmsNormForward(hX, hW, hY, hInv, rows, inner, 1e-5)
    cuda.RmsNormBackward(hX, hW, hdY, hInv, hdX, hdW, rows, inner)
    dw1 = cuda.GetMemory(hdW, inner)
    cuda.RmsNormBackward(hX, hW, hdY, hInv, hdX, hdW, rows, inner)
    dw2 = cuda.GetMemory(hdW, inner)
    np.testing.assert_array_equal(dw1, dw2)
    _, dw_ref = oracle.rmsnorm_layer_backward(x, w, dy, 1e-5)
    assert rel_err(dw1, dw_ref) < 1e-5
    for m in (hX, hW, hdY, hdX, hY, hInv, hdW):
        cuda.FreeMemory(m)


# either side of every change of the kernels' shape: pieces of 128 floats a warp, of 1024 a CTA, and the unaligned ones
EDGES = [4, 252, 256, 260, 512, 516, 768, 772, 1024, 1028, 2048, 2052, 4096, 4100, 1, 255, 257, 511, 513, 1023, 1025, 4095, 4097]


def layernorm(cuda, x, dy, eps):
    """y and dx of (rows, inner) through the function ids."""
    rows, inner = x.shape
    h = cuda.CreateLayerNorm(0, x.size, 1, rows, inner, eps)
    m = [cuda.AllocMemory(v) for v in (x, x.size, dy, x.size)]
    cuda.LayerNormForward(h, m[0], m[1])
    cuda.LayerNormBackward(h, m[1], m[2], m[3])
    out = [cuda.GetMemory(m[i], x.size).reshape(x.shape) for i in (1, 3)]
    for v in m:
        cuda.FreeMemory(v)
    cuda.FreeLayerNorm(h)
    return out


@pytest.mark.parametrize("inner", EDGES)
def test_rows_at_the_edges_of_the_shapes(cuda, inner):
    rng = np.random.default_rng(inner)
    rows, eps = 37, 1e-5
    x = rng.standard_normal((1, rows, inner)).astype(np.float32)
    dy = rng.standard_normal(x.shape).astype(np.float32)
    w = (1 + 0.2 * rng.standard_normal(inner)).astype(np.float32)
    y, dx = layernorm(cuda, x[0], dy[0], eps)
    y_ref, sd = oracle.layernorm_forward(x, eps)
    if inner > 1:      # one element: zero, and the backward a difference of equal numbers
        assert rel_err(y, y_ref[0]) < 1e-5
        assert rel_err(dx, oracle.layernorm_backward(y_ref, dy, sd, eps)[0]) < 1e-5
    m = [cuda.AllocMemory(v) for v in (x, w, dy, x.size, x.size, rows, inner)]
    cuda.RmsNormForward(m[0], m[1], m[3], m[5], rows, inner, eps)
    cuda.RmsNormBackward(m[0], m[1], m[2], m[5], m[4], m[6], rows, inner)
    y, dx, dw = cuda.GetMemory(m[3], x.size), cuda.GetMemory(m[4], x.size), cuda.GetMemory(m[6], inner)
    dx_ref, dw_ref = oracle.rmsnorm_layer_backward(x, w, dy, eps)
    assert rel_err(y, oracle.rmsnorm_layer_forward(x, w, eps)[0].ravel()) < 1e-5
    # at one element dx = dy w (1 / rms - x^2 / rms^3): a thousandth to a hundred-thousandth of its terms
    scale = np.abs(dx_ref).max() if inner > 1 else np.abs(dy * w / x).max()
    assert np.abs(dx - dx_ref.ravel()).max() / scale < 1e-5
    assert rel_err(dw, dw_ref) < 1e-5
    for v in m:
        cuda.FreeMemory(v)


@pytest.mark.parametrize("rows,inner", [(1184, 900), (1185, 900), (1184, 1024), (1185, 1024), (2500, 1024)])
def test_rmsnorm_backward_of_eight_pieces_either_side_of_one_cta_per_sm(cuda, rows, inner):
    rng = np.random.default_rng(rows)
    x, dy = (rng.standard_normal((rows, inner)).astype(np.float32) for _ in range(2))
    w = (1 + 0.2 * rng.standard_normal(inner)).astype(np.float32)
    m = [cuda.AllocMemory(v) for v in (x, w, dy, x.size, x.size, rows, inner)]
    cuda.RmsNormForward(m[0], m[1], m[3], m[5], rows, inner, 1e-5)
    cuda.RmsNormBackward(m[0], m[1], m[2], m[5], m[4], m[6], rows, inner)
    dx_ref, dw_ref = oracle.rmsnorm_layer_backward(x, w, dy, 1e-5)
    assert rel_err(cuda.GetMemory(m[4], x.size), dx_ref.ravel()) < 1e-5
    assert rel_err(cuda.GetMemory(m[6], inner), dw_ref) < 1e-5
    for v in m:
        cuda.FreeMemory(v)


@pytest.mark.parametrize("inner", [300, 768, 771, 2048])
def test_layernorm_quotients_are_those_of_a_division(cuda, inner):
    """Forward: rows of small multiples of 2^-10 that cancel in pairs have the mean 0 without a rounding, so y is x / stdev as a
    division rounds it.  Backward: dy times 2^70 takes the plain division instead of the reciprocal's quotients and changes nothing
    else (every operation before it is exact under a power of two): the same bits, 2^70 larger."""
    import torch
    from mycaffe_b200 import _lib
    rng = np.random.default_rng(inner)
    rows = 64
    half = rng.integers(-4096, 4097, (rows, inner // 2)).astype(np.float32) / 1024
    x = np.concatenate([half, -half, np.zeros((rows, inner % 2), np.float32)], 1)
    x = np.take(x, rng.permutation(inner), 1)
    t = torch.from_numpy(x).cuda()
    y, sd = torch.empty_like(t), torch.empty(rows, device="cuda")
    assert _lib.load().mca_layernorm_forward_f32(t.data_ptr(), y.data_ptr(), sd.data_ptr(), rows, inner, 1e-5, None) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(y.cpu().numpy(), x / sd.cpu().numpy()[:, None])
    dy = rng.standard_normal(x.shape).astype(np.float32)
    big = np.float32(2.0) ** 70
    np.testing.assert_array_equal(layernorm(cuda, x, dy, 1e-5)[1] * big, layernorm(cuda, x, dy * big, 1e-5)[1])


@pytest.mark.parametrize("inner", [300, 768, 771, 2048])
def test_layernorm_quotients_of_vanishing_numbers(cuda, inner):
    """Rows of small integers times 2^-80 .. 2^-143 and zeros of both signs: every sum is exact and the means are zero, so both
    directions are the one division, also where the remainder of a quotient is too small for a subnormal number."""
    import torch
    from mycaffe_b200 import _lib
    rng = np.random.default_rng(inner)
    rows, eps = 64, 1e-5
    unit = np.ldexp(np.float32(1), -80 - np.arange(rows))[:, None].astype(np.float32)
    half = rng.integers(-64, 65, (rows, inner // 2)).astype(np.float32)
    order, tail = rng.permutation(inner), np.zeros((rows, inner % 2), np.float32)
    x = np.take(np.concatenate([half * unit, -half * unit, tail], 1), order, 1)
    y = np.take(np.concatenate([rng.integers(-64, 65, half.shape).astype(np.float32)] * 2 + [tail], 1), order, 1)
    assert np.signbit(x[x == 0]).any() and not np.signbit(x[x == 0]).all()
    lib = _lib.load()
    tx, ty = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    out, sd = torch.empty_like(tx), torch.empty(rows, device="cuda")
    assert lib.mca_layernorm_forward_f32(tx.data_ptr(), out.data_ptr(), sd.data_ptr(), rows, inner, eps, None) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy().view(np.int32), (x / sd.cpu().numpy()[:, None]).view(np.int32))
    sd = rng.uniform(0.25, 4, rows).astype(np.float32)   # the halves of x cancel, those of y are equal: m1 = m2 = 0
    tsd = torch.from_numpy(sd).cuda()
    assert lib.mca_layernorm_backward_f32(ty.data_ptr(), tx.data_ptr(), tsd.data_ptr(), out.data_ptr(), rows, inner, eps, None) == 0
    torch.cuda.synchronize()
    denom = np.repeat(sd[:, None], inner, 1)
    denom.ravel()[:rows] += np.float32(eps)              # the first `rows` elements, as the reference divides them
    np.testing.assert_array_equal(out.cpu().numpy().view(np.int32), (x / denom).view(np.int32))


def test_layernorm_of_rows_that_are_not_finite(cuda):
    """An infinity makes its own row nan and leaves the others as they are; a row whose squares overflow has an infinite
    deviation and is zero, as the division by it is."""
    rng = np.random.default_rng(5)
    x = rng.standard_normal((16, 768)).astype(np.float32)
    dy = rng.standard_normal(x.shape).astype(np.float32)
    y0, dx0 = layernorm(cuda, x, dy, 1e-5)
    bad, bad_dy = x.copy(), dy.copy()
    bad[14, 5] = np.inf
    bad[13] *= np.float32(1e25)
    bad_dy[15, 7] = np.inf
    y, dx = layernorm(cuda, bad, bad_dy, 1e-5)
    assert np.isnan(y[14]).all() and (y[13] == 0).all() and not np.isfinite(dx[15]).any()
    np.testing.assert_array_equal(y[:13], y0[:13])
    np.testing.assert_array_equal(dx[:13], dx0[:13])


def test_raw_entry_points_reject_bad_arguments():
    from mycaffe_b200 import _lib, function_ids as ids
    lib = _lib.load()
    assert lib.mca_layernorm_forward_f32(None, None, None, 4, 8, 1e-5, None) == ids.ERROR_PARAM_NULL
    assert lib.mca_rmsnorm_forward_f32(None, None, None, None, 4, 8, 1e-5, None) == ids.ERROR_PARAM_NULL
    assert lib.mca_rmsnorm_backward_scratch_floats(768) >= 768


@pytest.mark.parametrize("case", ["ln", "ln3", "ln3B", "ln-blk"])
def test_layernorm_ids_match_the_reference_vectors(cuda, pico_ln, case):
    """ids 970 / 975 / 976 on the reference's own LayerNorm vectors (gpt-pico-ln*, epsilon 1e-10): y from x, and the
    gradient at x from the gradient at y."""
    g = lambda n: pico_ln[f"{case}/{n}"]
    x = g("x")
    outer, channels, inner = x.shape
    h = cuda.CreateLayerNorm(0, x.size, outer, channels, inner, 1e-10)
    hX, hY, hdY, hdX = cuda.AllocMemory(x), cuda.AllocMemory(x.size), cuda.AllocMemory(g("grad_1a_y")), cuda.AllocMemory(x.size)
    cuda.LayerNormForward(h, hX, hY)
    np.testing.assert_allclose(cuda.GetMemory(hY, x.size).reshape(x.shape), g("y"), atol=5e-7)
    cuda.LayerNormBackward(h, hY, hdY, hdX)
    assert rel_err(cuda.GetMemory(hdX, x.size).reshape(x.shape), g("grad_9_x")) < 1e-5
    for m in (hX, hY, hdY, hdX):
        cuda.FreeMemory(m)
    cuda.FreeLayerNorm(h)


@pytest.mark.parametrize("case", ["blk", "blk3", "blk3B"])
def test_block_layernorm_then_attention_matches_the_reference_vectors(cuda, pico_ln, case):
    """The reference's transformer-block vectors through the library: 1_x -> LAYERNORM_FWD -> 2_x_ln11 -> the
    attention layer with ATTN_FWD at its core -> 3_x_attn; back: grad_8_x_attn -> ATTN_BWD -> grad_9_ln1 ->
    LAYERNORM_BWD (+ the residual branch) -> grad_10_x.  The InnerProduct glue either side of the attention core is
    the C# layer's and is restated in numpy."""
    from gpu_util import Sdpa
    from helpers import PICO_BLOCK_CASES, csa_backward, csa_forward
    H = PICO_BLOCK_CASES[case]
    g = lambda n: pico_ln[f"{case}/{n}"]
    x = g("1_x")
    B, T, Cn = x.shape
    hL = cuda.CreateLayerNorm(0, x.size, B, T, Cn, 1e-10)
    hX, hY = cuda.AllocMemory(x), cuda.AllocMemory(x.size)
    cuda.LayerNormForward(hL, hX, hY)
    ln1 = cuda.GetMemory(hY, x.size).reshape(x.shape)
    np.testing.assert_allclose(ln1, g("2_x_ln11"), atol=5e-7)

    a = Sdpa(cuda, B, T, H, Cn // H, training=True)
    mask = oracle.causal_mask(T)
    attn = csa_forward(ln1, g("attn_weight"), g("attn_bias"), g("attn_proj_weight"), g("attn_proj_bias"), H,
                       lambda q, k, v: a.forward(q, k, v, mask))
    np.testing.assert_allclose(attn, g("3_x_attn"), atol=3e-7)
    d_ln1 = csa_backward(ln1, g("attn_weight"), g("attn_bias"), g("attn_proj_weight"), H, g("grad_8_x_attn"),
                         lambda q, k, v, dy: a.backward(dy))
    assert rel_err(d_ln1, g("grad_9_ln1")) < 1e-5
    hdY, hdX = cuda.AllocMemory(g("grad_9_ln1")), cuda.AllocMemory(x.size)
    cuda.LayerNormBackward(hL, hY, hdY, hdX)
    dx = cuda.GetMemory(hdX, x.size).reshape(x.shape) + g("grad_8_x")
    assert rel_err(dx, g("grad_10_x")) < 1e-5
    a.close()
    for m in (hX, hY, hdY, hdX):
        cuda.FreeMemory(m)
    cuda.FreeLayerNorm(hL)
