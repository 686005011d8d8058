"""Split-operand attention of fp32 handles far from unit magnitude: tensors, or one operand against another, whose products of scales
leave the fp32 range, with causal and key masks and an item whose every key is masked.  Against the fp64 oracle."""
import numpy as np
import pytest

import oracle
from gpu_util import Sdpa

pytestmark = pytest.mark.gpu


def close(a, ref, steps=8, rel=2e-5):
    # fp32 products summed in fp32: far below 2e-5 of the output's scale (test_fp32_tiles_gpu); below 2^-126 the results' own grid
    # is 2^-149, a few steps of it for the sums that are taken there
    ref = np.asarray(ref, np.float64)
    return np.isfinite(a).all() and np.abs(a - ref).max() <= rel * np.abs(ref).max() + steps * 2.0 ** -149


@pytest.mark.parametrize("D", [16, 64, 128])
@pytest.mark.parametrize("kind", ["causal", "keys"])
@pytest.mark.parametrize("mq,mk,mv,mdy", [
    (1, 1, 1e-20, 1),           # a small tensor
    (1, 1, 1e-33, 1),           # ... whose reciprocal scale over a row sum would be subnormal
    (1, 1, 1, 1e-35),
    (1e-20, 1e-20, 1, 1),       # logits of zero
    (1e-20, 1e20, 1, 1),        # logits of one from scales that are far apart
    (1e-10, 1e10, 1e-16, 1e-16),
    (1e-17, 1e17, 1e17, 1e-17),
    (1, 1, 1e-39, 1),           # subnormal numbers
])
def test_magnitudes(D, kind, mq, mk, mv, mdy):
    from mycaffe_b200 import CudaDnn
    cuda = CudaDnn(0)
    B, H, T = 2, 2, 130
    rng = np.random.default_rng(D)
    q, k, v, dy = ((m * rng.standard_normal((B, H, T, D))).astype(np.float32) for m in (mq, mk, mv, mdy))
    if kind == "causal":
        mask, mode = oracle.causal_mask(T), 1
    else:
        mask, mode = (rng.random((B, T)) > 0.3).astype(np.float32), 2
        mask[1] = 0
    # 128-wide heads: the split forward belongs to the inference handle under a key mask, the backward is the exact one
    train = D != 128 or kind == "causal"
    a = Sdpa(cuda, B, T, H, D, training=train)
    y = a.forward(q, k, v, mask, batch_mask=mode == 2)
    assert close(y, oracle.sdpa_forward(q, k, v, mask, mode, f64=True))
    if train and D != 128:
        # dQ and dK see delta = rowsum(dY o Y), where each of D elements of the fp32 Y is half a step off, times K or Q / sqrt(D)
        steps = 8 + 0.5 * np.sqrt(D) * np.abs(dy).max() * max(np.abs(q).max(), np.abs(k).max())
        # dS is split into fp16 halves (grid 2^-25) at 2^-19 |dY'| |V'| P.  The largest scale there is, 2^126, leaves subnormal V at
        # |V'| ~ 2^-4 instead of 2^12: dS ~ 2^-8 P, with P ~ 2^-7 over these rows 2^-10 of each element, so below 2^-9 of the result
        rel = 2.0 ** -9 if mv < 2.0 ** -126 else 2e-5
        for name, g, r in zip("qkv", a.backward(dy), oracle.sdpa_backward(q, k, v, dy, mask, mode, f64=True)):
            assert close(g, r, steps, rel), name
    a.close()
    cuda.Dispose()
