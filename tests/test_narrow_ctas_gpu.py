"""bf16 heads of 64: the CTAs that share an SM (128 rows against 64 rows a step in the backward, P in columns of its own in the
forward) at lengths around their tiles, every mask form, and logits that outgrow the softmax's reference point from tile to tile,
against the fp64 oracle.  P, dS and the results are bf16 (2^-9 relative each) and sums of them keep that: well below 2e-2 of scale."""
import numpy as np
import pytest

import oracle
from gpu_util import Sdpa, bf16_round
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 63, 64, 65, 127, 129, 192, 193, 449])
@pytest.mark.parametrize("mask_kind", ["causal", "none", "keys"])
def test_forward_and_backward_at_the_edges(T, mask_kind):
    from mycaffe_b200 import CudaDnn
    from mycaffe_b200 import function_ids as ids
    cuda = CudaDnn(0)
    rng = np.random.default_rng(T)
    B, H, D = 2, 3, 64
    q, k, v, dy = (bf16_round(rng.standard_normal((B, H, T, D)).astype(np.float32)) for _ in range(4))
    k = bf16_round((k * (1 + 8 * np.arange(T) / 449)[None, None, :, None]).astype(np.float32))   # later keys, larger logits
    mask = (rng.random((B, T)) > 0.3).astype(np.float32) if mask_kind == "keys" else None
    mode = {"causal": 3, "none": 0, "keys": 2}[mask_kind]
    a = Sdpa(cuda, B, T, H, D, training=True, dtype=ids.MCA_DTYPE_BF16, flags=ids.MCA_FLAG_CAUSAL_IMPLICIT if mode == 3 else 0)
    y = a.forward(q, k, v, mask, batch_mask=mode == 2)
    assert rel_err(y, oracle.sdpa_forward(q, k, v, mask, mode, f64=True)) < 2e-2
    # At T = 1 dQ and dK are zero: dP - delta is then the difference of two fp32 sums of the same D products (each within
    # D 2^-24 of the sum of their magnitudes), scaled by 1 / sqrt(D) and multiplied by K or Q.
    zero = 2 * D * 2.0 ** -24 * np.abs(dy * v).sum(-1).max() / np.sqrt(D) * max(np.abs(q).max(), np.abs(k).max())
    for name, g, r in zip("qkv", a.backward(dy), oracle.sdpa_backward(q, k, v, dy, mask, mode, f64=True)):
        assert np.isfinite(g).all(), name
        if np.abs(r).max() < 1e-6:
            assert np.abs(g).max() <= zero, name
        else:
            assert rel_err(g, r) < 2e-2, name
    a.close()
    cuda.Dispose()
