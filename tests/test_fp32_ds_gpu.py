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


def test_handles_share_one_workspace():
    """dS lives inside one backward: handles of one kernel index hold one workspace between them, none where dS is never passed on, and
    it goes with the last of them.  Backwards in another order than the forwards use it in turn."""
    import torch
    cuda = CudaDnn(0)
    used = lambda: -torch.cuda.mem_get_info()[0]
    B, H, T, D = 2, 16, 1024, 96
    ds, own = B * H * T * T * 4, B * H * T * (4 * 4 + D * 4)
    new = lambda *s: Sdpa(cuda, *s, training=True, dtype=ids.MCA_DTYPE_F32, flags=ids.MCA_FLAG_EXACT_FP32)
    new(B, T, H, D).close()                                   # the context's own allocations
    start, slack = used(), 32 << 20
    few = [new(1, 256, 2, D) for _ in range(32)]              # too little work for the two-kernel form
    assert used() - start < slack
    many = [new(B, T, H, D) for _ in range(4)]
    assert used() - start < ds + 4 * own + slack
    for a in few + many[1:]:
        a.close()
    small = new(8, 200, 16, D)
    rng = np.random.default_rng(0)
    cases = []
    for a, shape in ((many[0], (B, H, T, D)), (small, (8, 16, 200, D))):
        t = [rng.standard_normal(shape).astype(np.float32) for _ in range(4)]
        a.forward(*t[:3], oracle.causal_mask(shape[2]))
        cases.append((a, t))
    for a, t in cases + cases[:1]:
        for g, r in zip(a.backward(t[3]), oracle.sdpa_backward(*t, oracle.causal_mask(t[0].shape[2]), 1, f64=True)):
            assert rel_err(g, r) < 2e-5
    many[0].close()
    small.close()
    assert used() - start < slack
    cuda.Dispose()
