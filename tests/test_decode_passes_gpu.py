"""Decode steps of one to nine sequences: the padded passes of the streaming projections (3, 5, 6 and 7 sequences), rows that are
or are not shared by warps, splits with and without a combine pass, against the restated step over several tokens."""
import ctypes as C
import subprocess

import numpy as np
import pytest

import oracle
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 2, 3, 5, 6, 7, 8, 9])
@pytest.mark.parametrize("dim,hidden,n_heads,n_kv,seq", [(288, 768, 6, 6, 64), (256, 1032, 4, 2, 700)])
def test_steps_match_the_restated_model(B, dim, hidden, n_heads, n_kv, seq):
    from mycaffe_b200.llama2 import TransformerGpu
    rng = np.random.default_rng(B * 100 + dim)
    cfg = dict(dim=dim, hidden_dim=hidden, n_layers=2, n_heads=n_heads, n_kv_heads=n_kv, vocab_size=77, seq_len=seq)
    kv = dim // n_heads * n_kv
    g = lambda *sh: (0.08 * rng.standard_normal(sh)).astype(np.float32)
    w = {"rms_att_weight": 1 + g(2, dim), "rms_ffn_weight": 1 + g(2, dim), "rms_final_weight": 1 + g(dim),
         "token_embedding_table": rng.standard_normal((77, dim)).astype(np.float32), "wq": g(2, dim, dim), "wk": g(2, kv, dim),
         "wv": g(2, kv, dim), "wo": g(2, dim, dim), "w1": g(2, hidden, dim), "w2": g(2, dim, hidden), "w3": g(2, hidden, dim),
         "wcls": g(77, dim)}
    t = TransformerGpu(0, batch=B, use_graph=True)
    t.load_weights(cfg, w)
    kc, vc = (rng.standard_normal((2, B, seq, kv)).astype(np.float32) for _ in range(2))   # a context already in the caches
    t.key_cache.copy_(t._torch.from_numpy(kc))
    t.value_cache.copy_(t._torch.from_numpy(vc))
    pos = rng.integers(0, seq - 3, B)
    pos[0] = seq - 4
    for step in range(3):                                  # eager, then from the graph
        tok = rng.integers(0, 77, B)
        ref = oracle.llama_forward(cfg, w, kc, vc, list(tok), list(pos + step))
        assert rel_err(t.forward_batch(tok, pos + step), ref) < 1e-4
    assert rel_err(t.key_cache.cpu().numpy(), kc) < 1e-5   # the appended rows, and nothing else


HAMMER = r"""
#include <thread>
#include <vector>
using Fn = int (*)(void*, void*, int, int, int, void*, void*);
struct Call { void *x, *w, *out, *stream; int B, dim, error; };
extern "C" void hammer(Fn fn, Call* calls, int n_calls, int rounds) {
  std::vector<std::thread> threads;
  for (int i = 0; i < n_calls; ++i)
    threads.emplace_back([=] {
      Call& c = calls[i];
      for (int r = 0; r < rounds && c.error == 0; ++r) c.error = fn(c.x, c.w, 0, c.B, c.dim, c.out, c.stream);
    });
  for (auto& t : threads) t.join();
}
"""


class Call(C.Structure):
    _fields_ = [(n, C.c_void_p) for n in ("x", "w", "out", "stream")] + [(n, C.c_int) for n in ("B", "dim", "error")]


@pytest.mark.parametrize("B", [1, 2, 4, 8])
def test_threads_with_rows_of_different_lengths(B, tmp_path):
    """Host threads whose projections read rows of different lengths through the same kernels, on streams of their own: every launch is
    accepted."""
    import torch
    from mycaffe_b200 import _lib
    (tmp_path / "hammer.cpp").write_text(HAMMER)
    so = str(tmp_path / "hammer.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", str(tmp_path / "hammer.cpp"), "-o", so], check=True)
    hammer = C.CDLL(so).hammer
    hammer.restype = None
    rounds, keep, calls = 3000, [], (Call * 4)()
    for call, dim in zip(calls, (256, 1536, 512, 1024)):
        w, x, out = torch.zeros(dim, dim, device="cuda"), torch.ones(B, dim, device="cuda"), torch.zeros(B, dim, device="cuda")
        w[:, 3] = 1
        stream = torch.cuda.Stream()
        keep.append((w, x, out, stream))
        call.x, call.w, call.out, call.stream, call.B, call.dim = x.data_ptr(), w.data_ptr(), out.data_ptr(), stream.cuda_stream, B, dim
    torch.cuda.synchronize()
    hammer(C.cast(_lib.load().mca_decode_out_proj, C.c_void_p), calls, len(calls), rounds)
    torch.cuda.synchronize()
    assert [c.error for c in calls] == [0] * len(calls)
    for _, _, out, _ in keep:
        assert bool((out == rounds).all())
