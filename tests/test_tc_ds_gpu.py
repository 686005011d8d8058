"""The tensor-core backward where dS passes through memory: heads enough for that (128-wide bf16 and 64-wide split operands; the shapes here are
claims of test_ds_rules_cpu.py, but for split heads of 65 rows in test_backward, which form dS twice), lengths around its tiles and the
pairs of them that share a CTA, every mask form with fully masked rows, against the fp64 oracle; heads that go through the workspace in
parts; handles that share it."""
import numpy as np
import pytest

import oracle
from gpu_util import Sdpa, bf16_round
from helpers import rel_err
from mycaffe_b200 import CudaDnn
from mycaffe_b200 import function_ids as ids

pytestmark = pytest.mark.gpu


def handle(cuda, B, T, H, D, bf16, mode):
    return Sdpa(cuda, B, T, H, D, training=True, dtype=ids.MCA_DTYPE_BF16 if bf16 else ids.MCA_DTYPE_F32,
                flags=ids.MCA_FLAG_CAUSAL_IMPLICIT if mode == 3 else 0)


@pytest.mark.parametrize("T", [65, 129, 193, 320])
@pytest.mark.parametrize("bf16", [True, False])
@pytest.mark.parametrize("kind", ["causal", "none", "keys", "pairs"])
def test_backward(T, bf16, kind):
    cuda = CudaDnn(0)
    rng = np.random.default_rng(T)
    B, H, D = 8, 18, 128 if bf16 else 64
    cast = bf16_round if bf16 else (lambda a: a)
    q, k, v, dy = (cast(rng.standard_normal((B, H, T, D)).astype(np.float32)) for _ in range(4))
    mode = {"causal": 3, "none": 0, "keys": 2, "pairs": 1}[kind]
    mask = {"keys": (rng.random((B, T)) > 0.3), "pairs": (rng.random((T, T)) > 0.3)}.get(kind)
    mask = None if mask is None else mask.astype(np.float32)
    a = handle(cuda, B, T, H, D, bf16, mode)
    a.forward(q, k, v, mask, batch_mask=mode == 2)
    # bf16: P, dS and the results are rounded to 2^-9; split: fp32 sums of products of 22-bit halves, as the path's other tests
    for name, g, r in zip("qkv", a.backward(dy), oracle.sdpa_backward(q, k, v, dy, mask, mode, f64=True)):
        assert rel_err(g, r) < (2e-2 if bf16 else 2e-5), name
    a.close()
    cuda.Dispose()


def test_heads_in_parts():
    """16 causal heads of 10000 x 128 ask for 1.7 GB and get 1: two launches of each kernel, against the kernels that form dS twice
    (the raw entry point has no workspace).  Same products, same roundings, the sums in the same order: the same bits."""
    import torch
    from mycaffe_b200 import _lib
    cuda, lib = CudaDnn(0), _lib.load()
    H, T, D = 16, 10000, 128
    gen = torch.Generator("cuda").manual_seed(3)
    q, k, v, dy = (torch.randn(1, H, T, D, generator=gen, device="cuda").bfloat16() for _ in range(4))
    a = handle(cuda, 1, T, H, D, True, 3)
    host = lambda t: t.float().cpu().numpy()
    y = a.forward(host(q), host(k), host(v), None)
    got = a.backward(host(dy))
    a.close()
    y = torch.from_numpy(y).cuda().bfloat16()
    lse, delta = torch.empty(H * T, device="cuda"), torch.empty(H * T, device="cuda")
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    grads = [torch.empty_like(q) for _ in range(3)]
    y2 = torch.empty_like(q)
    p = lambda t: t.data_ptr()
    assert lib.mca_sdpa_forward_tc(p(q), p(k), p(v), ids.MCA_DTYPE_BF16, 1, 1, H, T, D, p(y2), p(lse), p(status), None) == 0
    assert lib.mca_sdpa_backward_tc(p(q), p(k), p(v), p(y), p(dy), p(lse), p(delta), ids.MCA_DTYPE_BF16, 1, 1, H, T, D, *map(p, grads), p(status), None) == 0
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    for g, r in zip(got, grads):
        assert np.array_equal(g, host(r))
    cuda.Dispose()


@pytest.mark.parametrize("T,B,H,bf16", [(2, 10, 26, False), (65, 10, 26, False), (128, 10, 26, False), (450, 4, 37, False), (450, 4, 37, True)])
@pytest.mark.parametrize("kind", ["causal", "none", "keys", "pairs"])
def test_one_tile_and_rows_without_a_key(T, B, H, bf16, kind):
    cuda = CudaDnn(0)
    rng = np.random.default_rng(T + 7)
    D = 128 if bf16 else 64
    cast = bf16_round if bf16 else (lambda a: a)
    q, k, v, dy = (cast(rng.standard_normal((B, H, T, D)).astype(np.float32)) for _ in range(4))
    mode = {"causal": 3, "none": 0, "keys": 2, "pairs": 1}[kind]
    mask = {"keys": (rng.random((B, T)) > 0.3), "pairs": (rng.random((T, T)) > 0.3)}.get(kind)
    if mask is not None:
        mask = mask.astype(np.float32)
        mask[0 if kind == "keys" else T // 2] = 0            # an item, a row that attends to nothing: uniform probabilities
    a = handle(cuda, B, T, H, D, bf16, mode)
    a.forward(q, k, v, mask, batch_mask=mode == 2)
    for name, g, r in zip("qkv", a.backward(dy), oracle.sdpa_backward(q, k, v, dy, mask, mode, f64=True)):
        assert rel_err(g, r) < (2e-2 if bf16 else 2e-5), name   # as in test_backward
    a.close()
    cuda.Dispose()


def test_handles_share_one_workspace():
    """Handles of either kind hold one workspace between them, it goes with the last of them, and one that never passes dS holds none; backwards
    in another order than the forwards use it in turn."""
    import torch
    cuda = CudaDnn(0)
    used = lambda: -torch.cuda.mem_get_info()[0]
    handle(cuda, 1, 512, 100, 64, False, 3).close()              # the context's own allocations
    start, slack = used(), 32 << 20
    room = 96 * 36 * 4 * 128 * 128                               # 96 heads, the lower triangle of 8 x 8 tiles, two halves of 2 bytes
    first = handle(cuda, 8, 1024, 12, 64, False, 3)
    one = used()
    second = handle(cuda, 8, 1024, 12, 64, False, 3)
    own = used() - one
    assert abs(one - start - own - room) < slack
    first.close()
    second.close()
    assert used() - start < slack
    none = handle(cuda, 1, 16384, 16, 128, True, 3)              # too few heads fit at a time: dS is formed twice
    assert used() - start < 16 * 16384 * (4 * 4 + 128 * 4) + slack
    none.close()
    rng = np.random.default_rng(0)
    cases = []
    for B, H, T, bf16, mode in ((8, 18, 320, False, 0), (8, 18, 193, True, 3), (8, 18, 200, False, 3)):
        cast = bf16_round if bf16 else (lambda a: a)
        t = [cast(rng.standard_normal((B, H, T, 128 if bf16 else 64)).astype(np.float32)) for _ in range(4)]
        a = handle(cuda, B, T, H, t[0].shape[3], bf16, mode)
        a.forward(*t[:3], None)
        cases.append((a, t, bf16, mode))
    for a, t, bf16, mode in cases + cases[:1]:
        for g, r in zip(a.backward(t[3]), oracle.sdpa_backward(*t, None, mode, f64=True)):
            assert rel_err(g, r) < (2e-2 if bf16 else 2e-5)
    for a, *_ in cases:
        a.close()
    assert used() - start < slack
    cuda.Dispose()


@pytest.mark.parametrize("bf16,B,H,T", [(False, 8, 8, 512), (True, 1, 16, 2048)])
def test_a_handle_does_not_see_the_room_of_others(bf16, B, H, T):
    """The gradients' bits are the same whether or not a handle that asked for more room exists."""
    cuda = CudaDnn(0)
    rng = np.random.default_rng(1)
    D = 128 if bf16 else 64
    t = [rng.standard_normal((B, H, T, D)).astype(np.float32) for _ in range(4)]
    got = []
    for alone in (True, False):
        other = None if alone else handle(cuda, 1, 4096, 32, D, bf16, 3)
        a = handle(cuda, B, T, H, D, bf16, 0)
        a.forward(*t[:3], None)
        got.append(a.backward(t[3]))
        a.close()
        if other:
            other.close()
    for g, r in zip(*got):
        assert np.array_equal(g, r)
    cuda.Dispose()
