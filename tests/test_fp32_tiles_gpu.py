"""The fp32 kernels at the edges of their tiles.  Exact ones: both row-tile heights (64 for few or short heads, 128 otherwise), head
sizes either side of every padded size, the walked side's remainder, and head sizes whose
rows are not 16-byte aligned (the copies that are not asynchronous).  Against the fp64 oracle."""
import numpy as np
import pytest

import oracle
from gpu_util import Sdpa
from helpers import rel_err
from mycaffe_b200 import function_ids as ids

pytestmark = pytest.mark.gpu

# fp32 products summed in fp32: about sqrt(T D) roundings of 2^-24 on terms of the output's scale, far below 2e-5 for T D < 1e6
TOL = 2e-5


@pytest.fixture(scope="module")
def cuda():
    from mycaffe_b200 import CudaDnn
    c = CudaDnn(0)
    yield c
    c.Dispose()


@pytest.mark.parametrize("B,H,T,D", [
    (1, 2, 65, 48), (1, 1, 193, 80), (2, 1, 127, 96), (1, 1, 129, 128),        # 64-row tiles
    (40, 4, 128, 32), (38, 4, 129, 64), (20, 8, 255, 48), (16, 10, 193, 96),   # 128-row tiles
    (25, 6, 200, 80), (19, 8, 190, 128), (40, 4, 130, 7), (1, 2, 66, 33), (2, 2, 64, 100)])
@pytest.mark.parametrize("kind", ["causal", "keys"])
def test_tiles_forward_backward(cuda, B, H, T, D, kind):
    rng = np.random.default_rng(B * 1000 + T * 10 + D)
    q, k, v, dy = (rng.standard_normal((B, H, T, D)).astype(np.float32) for _ in range(4))
    if kind == "causal":
        mask, mode = oracle.causal_mask(T), 1
    else:
        mask, mode = (rng.random((B, T)) > 0.3).astype(np.float32), 2
    a = Sdpa(cuda, B, T, H, D, training=True, dtype=ids.MCA_DTYPE_F32, flags=ids.MCA_FLAG_EXACT_FP32)
    y = a.forward(q, k, v, mask, batch_mask=mode == 2)
    got = a.backward(dy)
    a.close()
    assert rel_err(y, oracle.sdpa_forward(q, k, v, mask, mode, f64=True)) < TOL
    for g, r in zip(got, oracle.sdpa_backward(q, k, v, dy, mask, mode, f64=True)):
        assert rel_err(g, r) < TOL


@pytest.mark.parametrize("T,D", [(127, 64), (257, 32), (513, 64), (1025, 64), (2049, 16), (1100, 64)])
def test_split_operand_scales_per_head(cuda, T, D):
    """The operand split's scale belongs to a (batch, head): heads nine orders of magnitude apart keep their own precision, at every
    number of CTAs a head is spread over and where a head outgrows the registers it is kept in."""
    rng = np.random.default_rng(T + D)
    B, H = 1, 3
    mag = np.array([1e-5, 1.0, 3e3], np.float32).reshape(1, H, 1, 1)
    q, k, v, dy = (rng.standard_normal((B, H, T, D)).astype(np.float32) for _ in range(4))
    v, dy = v * mag, dy * mag[:, ::-1]
    q, k = q * np.array([1e-4, 1.0, 1e3], np.float32).reshape(1, H, 1, 1), k * np.array([1e4, 1.0, 1e-3], np.float32).reshape(1, H, 1, 1)
    mask = oracle.causal_mask(T)
    a = Sdpa(cuda, B, T, H, D, training=True)
    y = a.forward(q, k, v, mask)
    got = a.backward(dy)
    a.close()
    ref_y, ref = oracle.sdpa_forward(q, k, v, mask, 1, f64=True), oracle.sdpa_backward(q, k, v, dy, mask, 1, f64=True)
    for h in range(H):
        assert rel_err(y[:, h], ref_y[:, h]) < TOL
        for g, r in zip(got, ref):
            assert rel_err(g[:, h], r[:, h]) < TOL
