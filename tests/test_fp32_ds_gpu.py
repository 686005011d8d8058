"""The exact fp32 backward where dS passes through memory: enough heads for that, 64- and 128-row key tiles, query and key blocks
that end inside a tile, an odd number of query blocks, rows that are not 16-byte aligned.  Against the fp64 oracle."""
import numpy as np
import pytest

import oracle
from gpu_util import Sdpa
from helpers import rel_err
from mycaffe_b200 import CudaDnn
from mycaffe_b200 import function_ids as ids

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,T,D", [(10, 10, 129, 80), (8, 16, 65, 128), (25, 6, 193, 128), (30, 6, 257, 100), (20, 10, 150, 7)])
@pytest.mark.parametrize("kind", ["causal", "none", "keys"])
def test_backward(B, H, T, D, kind):
    cuda = CudaDnn(0)
    rng = np.random.default_rng(T + D)
    q, k, v, dy = (rng.standard_normal((B, H, T, D)).astype(np.float32) for _ in range(4))
    mask, mode = {"causal": (oracle.causal_mask(T), 1), "none": (None, 0),
                  "keys": ((rng.random((B, T)) > 0.3).astype(np.float32), 2)}[kind]
    a = Sdpa(cuda, B, T, H, D, training=True, dtype=ids.MCA_DTYPE_F32, flags=ids.MCA_FLAG_EXACT_FP32)
    a.forward(q, k, v, mask, batch_mask=mode == 2)
    # fp32 products summed in fp32: about sqrt(T D) roundings of 2^-24 on terms of the output's scale, far below 2e-5 for T D < 1e6
    for g, r in zip(a.backward(dy), oracle.sdpa_backward(q, k, v, dy, mask, mode, f64=True)):
        assert rel_err(g, r) < 2e-5
    a.close()
    cuda.Dispose()
