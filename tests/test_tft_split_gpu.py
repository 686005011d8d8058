"""TFT attention with few batch items: the heads and row tiles of an item over a cluster of CTAs, against the fp64 oracle at the
bound of the unsplit kernels (the same sums, the head sums and the tiles' parts in another fixed order)."""
import ctypes as C
import subprocess

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


def forward_and_backward(cuda, B, H, Nq, Nk, d, with_attn_grad, with_mask):
    rng = np.random.default_rng(B * 100 + H + Nq)
    q = rng.standard_normal((B, H, Nq, d)).astype(np.float32)
    k = rng.standard_normal((B, H, Nk, d)).astype(np.float32)
    v = rng.standard_normal((B, Nk, d)).astype(np.float32)
    mask = (np.arange(Nk)[None, :] > np.arange(Nq)[:, None] + Nk - Nq).astype(np.float32) if with_mask else None
    d_out = rng.standard_normal((B, Nq, d)).astype(np.float32)
    d_attn = rng.standard_normal((B, Nq, Nk)).astype(np.float32) if with_attn_grad else None
    h = [0 if a is None else cuda.AllocMemory(a) for a in (q, k, v, mask, d_out, d_attn)]
    o = [cuda.AllocMemory(n) for n in (B * Nq * d, B * Nq * Nk, q.size, k.size, v.size)]
    got = []
    for _ in range(2):
        cuda.TftAttnForward(h[0], h[1], h[2], h[3], B, H, Nq, Nk, d, o[0], o[1])
        cuda.TftAttnBackward(h[0], h[1], h[2], h[3], h[4], h[5], B, H, Nq, Nk, d, o[2], o[3], o[4])
        got.append([cuda.GetMemory(m, n) for m, n in zip(o, (B * Nq * d, B * Nq * Nk, q.size, k.size, v.size))])
    ref = [*oracle.tft_forward(q, k, v, mask, f64=True), *oracle.tft_backward(q, k, v, mask, d_out, d_attn, f64=True)]
    for a, b, r in zip(*got, ref):
        assert rel_err(a, np.ravel(r)) < 2e-5
        np.testing.assert_array_equal(a, b)          # whichever CTA came first
    for m in h + o:
        if m:
            cuda.FreeMemory(m)


# heads that are no multiple of the CTAs along them, row tiles likewise, a last tile of one row, one head, one tile, every head size of
# the backward; the forward (64-wide heads of 116 keys or more, else generic) over 1, 2, 4 and 8 CTAs: test_tft_rules_cpu.py
FORWARDS = [(1, 3, 49, 191, 64), (33, 6, 24, 192, 64), (2, 8, 30, 116, 64), (160, 4, 24, 120, 64), (2, 8, 24, 115, 64)]


@pytest.mark.parametrize("with_attn_grad", [False, True])
@pytest.mark.parametrize("B,H,Nq,Nk,d", [(2, 8, 24, 60, 32), (3, 4, 60, 60, 16), (2, 1, 100, 100, 64), (2, 5, 50, 70, 32), (1, 3, 49, 191, 64),
                                         (16, 8, 160, 160, 32), (2, 7, 25, 33, 64), (40, 2, 73, 90, 16), (33, 6, 24, 192, 64)] + FORWARDS[2:])
def test_split_over_a_cluster(cuda, B, H, Nq, Nk, d, with_attn_grad):
    forward_and_backward(cuda, B, H, Nq, Nk, d, with_attn_grad, with_mask=True)


@pytest.mark.parametrize("B,H,Nq,Nk,d", FORWARDS)
def test_split_without_a_mask(cuda, B, H, Nq, Nk, d):
    forward_and_backward(cuda, B, H, Nq, Nk, d, with_attn_grad=False, with_mask=False)


@pytest.mark.parametrize("B,H,Nq,Nk,d", [(140, 2, 100, 60, 64), (130, 1, 190, 33, 32), (150, 3, 90, 17, 16), (140, 1, 120, 192, 64)])
def test_row_tiles_of_one_cta(cuda, B, H, Nq, Nk, d):
    """Items that fill the chip: one CTA walks an item's row tiles and asks for the next tile's rows while it works on this one's.  They
    must not land where a slower warp still reads: every one of many runs gives the bits of the first, and the first is the oracle's."""
    import torch
    from mycaffe_b200 import _lib
    rng = np.random.default_rng(B + Nk)
    q, k, v, go = (rng.standard_normal(s).astype(np.float32) for s in ((B, H, Nq, d), (B, H, Nk, d), (B, Nk, d), (B, Nq, d)))
    t = [torch.from_numpy(a).cuda() for a in (q, k, v, go)]
    o = [torch.empty_like(a) for a in t[:3]]
    first = None
    for _ in range(25):
        for a in o:
            a.fill_(float("nan"))
        assert _lib.load().mca_tft_attention_backward_f32(*(a.data_ptr() for a in t[:3]), None, t[3].data_ptr(), None, B, H, Nq, Nk, d,
                                                          *(a.data_ptr() for a in o), torch.cuda.current_stream().cuda_stream) == 0
        if first is None:
            first = [a.clone() for a in o]
            for a, r in zip(first, oracle.tft_backward(q, k, v, None, go, None, f64=True)):
                assert rel_err(a.cpu().numpy(), r) < 2e-5
        assert all(torch.equal(a, b) for a, b in zip(o, first))


@pytest.mark.parametrize("B,H,Nq,Nk", [(1, 3, 49, 191), (2, 2, 30, 120)])
def test_queries_without_16_byte_alignment(cuda, B, H, Nq, Nk):
    """A caller of the C entry point may hand in q at any float; at these shapes the same call with an aligned q takes the tiled kernel."""
    import torch
    from mycaffe_b200 import _lib
    rng = np.random.default_rng(Nk)
    d = 64
    q, k, v = (rng.standard_normal(s).astype(np.float32) for s in ((B, H, Nq, d), (B, H, Nk, d), (B, Nk, d)))
    room = torch.zeros(q.size + 4, device="cuda")
    tk, tv = torch.from_numpy(k).cuda(), torch.from_numpy(v).cuda()
    out, attn = torch.empty(B * Nq * d, device="cuda"), torch.empty(B * Nq * Nk, device="cuda")
    ref = oracle.tft_forward(q, k, v, None, f64=True)
    for offset in (0, 1, 2, 3):
        tq = room[offset:offset + q.size]
        tq.copy_(torch.from_numpy(q.ravel()))
        assert _lib.load().mca_tft_attention_forward_f32(tq.data_ptr(), tk.data_ptr(), tv.data_ptr(), None, B, H, Nq, Nk, d, out.data_ptr(),
                                                         attn.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        assert rel_err(out.cpu().numpy(), np.ravel(ref[0])) < 2e-5
        assert rel_err(attn.cpu().numpy(), np.ravel(ref[1])) < 2e-5


HAMMER = r"""
#include <thread>
#include <vector>
using Fwd = int (*)(void*, void*, void*, void*, int, int, int, int, int, void*, void*, void*);
using Bwd = int (*)(void*, void*, void*, void*, void*, void*, int, int, int, int, int, void*, void*, void*, void*);
struct Call { void* p[10]; int n[5]; int error; };   // q k v d_out | out attn dq dk dv | stream;  B H Nq Nk d
extern "C" void hammer(Fwd fwd, Bwd bwd, Call* calls, int n_calls, int rounds) {
  std::vector<std::thread> threads;
  for (int i = 0; i < n_calls; ++i)
    threads.emplace_back([=] {
      Call& c = calls[i];
      void* const* p = c.p;
      const int* n = c.n;
      for (int r = 0; r < rounds && c.error == 0; ++r) {
        c.error = fwd(p[0], p[1], p[2], nullptr, n[0], n[1], n[2], n[3], n[4], p[4], p[5], p[9]);
        if (c.error == 0) c.error = bwd(p[0], p[1], p[2], nullptr, p[3], nullptr, n[0], n[1], n[2], n[3], n[4], p[6], p[7], p[8], p[9]);
      }
    });
  for (auto& t : threads) t.join();
}
"""


class Call(C.Structure):
    _fields_ = [("p", C.c_void_p * 10), ("n", C.c_int * 5), ("error", C.c_int)]


def test_threads_with_different_sizes(cuda, tmp_path):
    """Host threads that call the C entry points on streams of their own, some with long key rows and some with short ones: every launch
    is accepted and every result is the one of the calls made alone."""
    import torch
    from mycaffe_b200 import _lib
    (tmp_path / "hammer.cpp").write_text(HAMMER)
    so = str(tmp_path / "hammer.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", str(tmp_path / "hammer.cpp"), "-o", so], check=True)
    lib, hammer = _lib.load(), C.CDLL(so).hammer
    hammer.restype = None
    fwd, bwd = (C.cast(f, C.c_void_p) for f in (lib.mca_tft_attention_forward_f32, lib.mca_tft_attention_backward_f32))
    B, H, Nq = 2, 2, 30
    shapes = [(192, 64), (117, 64), (40, 32), (190, 32)]          # tiled and generic forwards, long and short rows of each
    calls, outputs, keep = (Call * len(shapes))(), [], []
    for call, (Nk, d) in zip(calls, shapes):
        g = torch.Generator(device="cuda").manual_seed(Nk)
        ins = [torch.randn(s, generator=g, device="cuda") for s in ((B, H, Nq, d), (B, H, Nk, d), (B, Nk, d), (B, Nq, d))]
        outs = [torch.empty(s, device="cuda") for s in ((B, Nq, d), (B, Nq, Nk), (B, H, Nq, d), (B, H, Nk, d), (B, Nk, d))]
        keep.append((ins, torch.cuda.Stream()))
        outputs.append(outs)
        call.p[:] = [t.data_ptr() for t in ins + outs] + [keep[-1][1].cuda_stream]
        call.n[:] = [B, H, Nq, Nk, d]
    torch.cuda.synchronize()
    alone = []
    for i, outs in enumerate(outputs):
        hammer(fwd, bwd, C.byref(calls[i]), 1, 1)
        torch.cuda.synchronize()
        alone.append([t.clone() for t in outs])
    hammer(fwd, bwd, calls, len(shapes), 3000)
    torch.cuda.synchronize()
    assert [c.error for c in calls] == [0] * len(shapes)
    for outs, want in zip(outputs, alone):
        assert all(torch.equal(a, b) for a, b in zip(outs, want))
