"""The one-launch fp32 forward of short inference calls: lengths around its 32-key steps and its rows per warp, one to three CTAs a
head, every mask form with fully masked rows, the packed layout, and the calls beyond its rule, against the fp64 oracle."""
import numpy as np
import pytest

import oracle
from gpu_util import Sdpa
from helpers import rel_err
from mycaffe_b200 import CudaDnn
from mycaffe_b200 import function_ids as ids

pytestmark = pytest.mark.gpu

# fp32 dot products of up to 64 terms and sums of up to 128 probabilities (about sqrt(n) 2^-24 each), ex2 and a division at 2^-22
TOL = 3e-6


@pytest.mark.parametrize("T", [1, 2, 31, 33, 64, 97, 127, 128, 129])
@pytest.mark.parametrize("B,H,D", [(1, 1, 16), (1, 5, 32), (2, 9, 64), (4, 9, 16), (3, 16, 64)])
def test_forward(T, B, H, D):
    cuda = CudaDnn(0)
    rng = np.random.default_rng(T * 100 + D)
    q, k, v = (2 * rng.standard_normal((B, H, T, D)).astype(np.float32) for _ in range(3))
    keys = (rng.random((B, T)) > 0.3).astype(np.float32)
    keys[0] = 0                                            # every key masked: a uniform row
    pairs = (rng.random((T, T)) > 0.3).astype(np.float32)
    pairs[T // 2] = 0
    for mask, mode in ((None, 0), (oracle.causal_mask(T), 1), (pairs, 1), (keys, 2), (None, 3)):
        a = Sdpa(cuda, B, T, H, D, flags=ids.MCA_FLAG_CAUSAL_IMPLICIT if mode == 3 else 0, dtype=ids.MCA_DTYPE_F32)
        y = a.forward(q, k, v, mask, batch_mask=mode == 2)
        # past 128 keys the split-operand kernels take the call: their bound
        assert rel_err(y, oracle.sdpa_forward(q, k, v, mask, mode, f64=True)) < (TOL if T <= 128 else 2e-5), mode
        a.close()
    cuda.Dispose()


@pytest.mark.parametrize("T,H,D", [(50, 3, 64), (128, 4, 16)])
def test_packed(T, H, D):
    cuda = CudaDnn(0)
    rng = np.random.default_rng(T)
    B = 2
    x = rng.standard_normal((B, T, 3, H, D)).astype(np.float32)
    hc, ha = cuda.CreateCuDNN(), cuda.CreateAttn()
    cuda.SetAttn(hc, ha, 0, False, B, T, H, D, 0.0, 0, ids.MCA_DTYPE_F32, ids.MCA_FLAG_CAUSAL_IMPLICIT)
    hx, hy = cuda.AllocMemory(x), cuda.AllocMemory(B * T * H * D)
    cuda.AttnScaledDotProductForwardPacked(hc, ha, T, hx, 0, hy, False)
    y = cuda.GetMemory(hy, B * T * H * D).reshape(B, T, H, D).transpose(0, 2, 1, 3)
    q, k, v = (np.ascontiguousarray(x[:, :, i].transpose(0, 2, 1, 3)) for i in range(3))
    assert rel_err(y, oracle.sdpa_forward(q, k, v, None, 3, f64=True)) < TOL
    cuda.Dispose()


@pytest.mark.parametrize("over", ["q", "k", "v", "mask"])
@pytest.mark.parametrize("T,H,D", [(128, 4, 64), (100, 9, 32)])
def test_output_over_an_input(T, H, D, over):
    """y may be q's, k's, v's or the mask's memory: the split kernels take such a call, which read all of them before they write."""
    cuda = CudaDnn(0)
    rng = np.random.default_rng(T)
    q, k, v = (rng.standard_normal((1, H, T, D)).astype(np.float32) for _ in range(3))
    pairs = (rng.random((T, T)) > 0.3).astype(np.float32)
    hc, ha = cuda.CreateCuDNN(), cuda.CreateAttn()
    cuda.SetAttn(hc, ha, 0, False, 1, T, H, D, 0.0, 0, ids.MCA_DTYPE_F32, 0)
    room = np.zeros(max(T * T, q.size), np.float32)
    room[:T * T] = pairs.ravel()
    h = {"q": cuda.AllocMemory(q), "k": cuda.AllocMemory(k), "v": cuda.AllocMemory(v), "mask": cuda.AllocMemory(room)}
    cuda.AttnScaledDotProductForward(hc, ha, T, h["q"], h["k"], h["v"], h["mask"], h[over], False)
    y = cuda.GetMemory(h[over], q.size).reshape(q.shape)
    assert rel_err(y, oracle.sdpa_forward(q, k, v, pairs, 1, f64=True)) < 2e-5     # the split kernels' bound
    cuda.Dispose()
