"""Kernels that are let go early, late or not before the one ahead has ended (launch_rules.h), forwards with an SM for each CTA and with more CTAs, and
short forwards: calls in a row that nobody waits for give the bits of calls that are waited for one by one, over alternating inputs."""
import numpy as np
import pytest

from gpu_util import Sdpa
from mycaffe_b200 import CudaDnn
from mycaffe_b200 import function_ids as ids

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16,D,H,T,kind,train", [
    (True, 64, 7, 358, "keys", True), (True, 64, 40, 200, "keys", True), (True, 128, 5, 300, "keys", True), (True, 128, 11, 600, "pairs", True),
    (True, 64, 9, 520, "causal", True), (True, 64, 16, 600, "causal", True), (True, 64, 10, 900, "none", True),
    (False, 64, 12, 1100, "keys", True), (False, 32, 37, 512, "none", False), (False, 64, 38, 500, "pairs", True),
    (False, 32, 24, 128, "keys", False), (False, 64, 17, 100, "causal", False)])
def test_calls_in_a_row(bf16, D, H, T, kind, train):
    rng = np.random.default_rng(T)
    mask = {"keys": rng.random((1, T)) > 0.3, "pairs": rng.random((T, T)) > 0.3}.get(kind)
    data = [[rng.standard_normal((1, H, T, D)).astype(np.float32) for _ in range(4)] for _ in range(2)]
    results = []
    for asynchronous in (False, True):
        cuda = CudaDnn(0)
        cuda.SetAsync(asynchronous)
        a = Sdpa(cuda, 1, T, H, D, training=train, dtype=ids.MCA_DTYPE_BF16 if bf16 else ids.MCA_DTYPE_F32,
                 flags=ids.MCA_FLAG_CAUSAL_IMPLICIT if kind == "causal" else 0)
        hm = 0 if mask is None else cuda.AllocMemory(mask.astype(np.float32))
        inputs = [[a._alloc(x) for x in d] for d in data]
        outputs = [[a._alloc(data[0][0].size) for _ in range(4)] for _ in data]
        for _ in range(3):
            for (q, k, v, dy), (y, dq, dk, dv) in zip(inputs, outputs):
                cuda.AttnScaledDotProductForward(a.hCudnn, a.hAttn, T, q, k, v, hm, y, kind == "keys")
                if train:
                    cuda.AttnScaledDotProductBackward(a.hCudnn, a.hAttn, q, dq, k, dk, v, dv, 0, y, dy)
        cuda.SynchronizeDevice()
        results.append([cuda.GetMemory(h, data[0][0].size) for o in outputs for h in (o if train else o[:1])])
        a.close()
        if hm:
            cuda.FreeMemory(hm)
        cuda.Dispose()
    for g, r in zip(*results):
        assert np.any(r) and np.array_equal(g, r)
