"""The measured cases of this library: what a host program has it do, through the calls such a program makes.

Attention, decode, TFT and norm cases go through ``CudaDnn`` (function ids and memory handles, as MyCaffe's layers do), the
whole-token cases through ``TransformerGpu`` and ``mca_llama_forward``.  Inputs are made on the GPU from the seed.
"""
import ctypes as C
import math

import numpy as np
import torch

from mycaffe_b200 import CudaDnn, _lib
from mycaffe_b200 import function_ids as ids
from mycaffe_b200 import llama2

# --------------------------------------------------------------------------------------------------------------- cases


def attn(name, B, H, T, D, dtype="f32", mask="handle", train=True, packed=False, asynchronous=False):
    """One attention layer's core.  mask: "handle" = the lower-triangular (T,T) tensor CausalSelfAttentionLayer passes,
    "flag" = the handle's analytic causal flag, "key" = a (B,T) key mask as MultiheadAttentionLayer passes.  train: forward
    and backward, else the forward alone.  packed: q, k, v as the thirds of the c_attn output.  asynchronous: the calls
    do not wait for the GPU (the default is that each does, as the reference's)."""
    return dict(name=name, kind="attn", B=B, H=H, T=T, D=D, dtype=dtype, mask=mask, train=train, packed=packed,
                asynchronous=asynchronous)


def decode(name, B, H, kv, hs, seq, bf16, asynchronous):
    return dict(name=name, kind="decode", B=B, H=H, kv=kv, hs=hs, seq=seq, bf16=bf16, asynchronous=asynchronous)


def token(name, B, layers, heads, hs, hidden, vocab, seq, bf16):
    return dict(name=name, kind="token", B=B, layers=layers, heads=heads, hs=hs, hidden=hidden, vocab=vocab, seq=seq, bf16=bf16)


def step(name, B, layers, heads, kv, hidden, vocab, seq, bf16):
    return dict(name=name, kind="step", B=B, layers=layers, heads=heads, kv=kv, hs=128, hidden=hidden, vocab=vocab, seq=seq,
                bf16=bf16)


def tft(name, B, H, Nq, Nk, d, asynchronous):
    return dict(name=name, kind="tft", B=B, H=H, Nq=Nq, Nk=Nk, d=d, asynchronous=asynchronous)


def norm(name, op, rows, inner, asynchronous):
    """op: "layernorm" or "rmsnorm" of (rows, inner); forward and backward."""
    return dict(name=name, kind="norm", op=op, rows=rows, inner=inner, asynchronous=asynchronous)


def listed():
    return [
        # the smallest call: one causal self-attention block at inference (4 heads x 16, 128 tokens)
        attn("block_forward_small", 1, 4, 128, 16, train=False),
        # GPT training, the attention core of one GPT-2-small layer, as an unmodified C# layer calls it
        attn("gpt_train_f32", 8, 12, 1024, 64),
        # the same layer in bf16 from the packed c_attn output, with the causal flag, the calls not waiting
        attn("gpt_train_bf16", 8, 12, 1024, 64, dtype="bf16", mask="flag", packed=True, asynchronous=True),
        # encoder / cross-attention training under a key mask: the shape of the reference's own timing test
        attn("mha_key_mask_train", 3, 8, 200, 64, mask="key"),
        # training with wide fp32 heads at a length that is no multiple of a tile
        attn("wide_head_train_f32", 2, 16, 1500, 128),
        # long-context prefill, the headline shape for one sequence
        attn("prefill_32k_bf16", 1, 16, 32768, 128, dtype="bf16", mask="flag", train=False, asynchronous=True),
        # long-context training in bf16, an odd length
        attn("train_7001_bf16", 1, 16, 7001, 128, dtype="bf16", mask="flag", asynchronous=True),
        # KV-cache decode attention of a llama2-7B layer, 64 sequences of ragged length
        decode("decode_64_sequences", 64, 32, 32, 128, 4096, False, False),
        # text generation for one user: a whole token of a llama2.c 110M model, host call to host logits
        token("token_110m", 1, 12, 12, 64, 2048, 32000, 1024, False),
        # serving: a decode step of 16 sequences through 7B-shaped layers (four of them and the classifier), bf16
        step("serve_16_sequences", 16, 4, 32, 32, 11008, 32000, 2048, True),
        # TFT interpretable attention training (24 decoder steps over 192)
        tft("tft_train", 256, 4, 24, 192, 64, False),
        # LayerNorm of a GPT-2-small block, forward and backward
        norm("layernorm_gpt2", "layernorm", 8192, 768, False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a family, then sizes over the range the listed cases stand for."""
    family = rng.choice(["block", "gpt_f32", "gpt_bf16", "mha", "wide_f32", "prefill", "long_bf16", "decode", "token", "step", "tft",
                         "norm"])
    wait_not = rng.random() < 0.5
    if family == "block":          # a short forward
        c = attn("", rng.randint(1, 4), rng.randint(1, 16), _log(rng, 16, 1024), rng.choice([16, 32, 64]), train=False,
                 mask=rng.choice(["handle", "flag", "key"]), packed=rng.random() < 0.3, asynchronous=wait_not)
    elif family == "gpt_f32":      # head sizes of small GPT models, 48 (llama2.c) among them
        c = attn("", _log(rng, 1, 16), rng.randint(4, 16), _log(rng, 64, 2048), rng.choice([16, 32, 48, 64, 64, 64]),
                 mask=rng.choice(["handle", "flag"]), packed=rng.random() < 0.5, asynchronous=wait_not)
    elif family == "gpt_bf16":
        c = attn("", _log(rng, 1, 16), rng.randint(4, 16), _log(rng, 64, 2048), rng.choice([64, 64, 128]), dtype="bf16",
                 mask=rng.choice(["handle", "flag"]), packed=rng.random() < 0.5, asynchronous=wait_not)
    elif family == "mha":
        dtype = rng.choice(["f32", "f32", "bf16"])
        c = attn("", _log(rng, 1, 16), rng.randint(4, 16), _log(rng, 32, 1024), 64 if dtype == "bf16" else rng.choice([32, 64]),
                 dtype=dtype, mask="key", asynchronous=wait_not)
    elif family == "wide_f32":     # 80 and 96: head sizes of larger GPT models
        c = attn("", rng.randint(1, 2), rng.randint(4, 16), _log(rng, 128, 2048), rng.choice([80, 96, 128, 128]),
                 mask=rng.choice(["handle", "flag"]), packed=rng.random() < 0.3, asynchronous=wait_not)
    elif family == "prefill":
        D, T = rng.choice([64, 128, 128]), _log(rng, 1024, 32768)
        c = attn("", rng.randint(1, 4 if T < 16384 else 1), rng.randint(8, 16), T, D, dtype="bf16", mask="flag", train=False,
                 packed=rng.random() < 0.3, asynchronous=True)
    elif family == "long_bf16":
        c = attn("", 1, rng.randint(8, 16), _log(rng, 2048, 10000), rng.choice([64, 128]), dtype="bf16",
                 mask=rng.choice(["handle", "flag"]), packed=rng.random() < 0.3, asynchronous=True)
    elif family == "decode":
        H = rng.choice([8, 16, 32])
        c = decode("", _log(rng, 1, 64), H, rng.choice([H, H, H // 4]), rng.choice([48, 64, 96, 128, 128]), _log(rng, 256, 4096),
                   rng.random() < 0.5, wait_not)
    elif family == "token":
        heads, hs = rng.randint(6, 12), rng.choice([48, 64])
        c = token("", _log(rng, 1, 8), rng.randint(6, 12), heads, hs, 8 * rng.randint(heads * hs // 4, heads * hs // 3), 32000,
                  rng.choice([256, 512, 1024]), rng.random() < 0.3)
    elif family == "step":
        heads = rng.choice([16, 24, 32])
        c = step("", _log(rng, 1, 64), rng.randint(1, 4), heads, rng.choice([heads, heads // 4]), 64 * rng.randint(4 * heads, 5 * heads),
                 32000, _log(rng, 256, 2048), rng.random() < 0.5)
    elif family == "tft":
        Nk = rng.randint(32, 192)
        c = tft("", _log(rng, 16, 256), rng.choice([1, 2, 4, 8]), rng.choice([max(1, Nk // 8), rng.randint(1, Nk), Nk]), Nk,
                rng.choice([16, 32, 64]), wait_not)
    else:
        inner = _log(rng, 48, 4096)
        c = norm("", rng.choice(["layernorm", "rmsnorm"]), _log(rng, 64, 16384), inner if rng.random() < 0.25 else max(16, inner // 16 * 16),
                 wait_not)
    del c["name"]
    return c


# ---------------------------------------------------------------------------------------------------- preparing a state


class _Handle:
    """A memory handle seen as a torch tensor without a copy; keeps its CudaDnn (which owns the memory) alive."""

    def __init__(self, cuda, handle, shape, bf16):
        self.cuda = cuda
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr="<i2" if bf16 else "<f4",
                                             data=(cuda.GetPointer(handle), False), version=3)


class _Memory:
    """Memory handles of one CudaDnn with their torch views."""

    def __init__(self, seed, asynchronous):
        self.cuda = CudaDnn(0)
        self.cuda.SetAsync(asynchronous)
        self.gen = torch.Generator("cuda").manual_seed(int(seed))

    def empty(self, shape, bf16=False):
        h = (self.cuda.AllocMemoryBf16 if bf16 else self.cuda.AllocMemory)(int(np.prod(shape)))
        t = torch.as_tensor(_Handle(self.cuda, h, shape, bf16), device="cuda")
        return h, t.view(torch.bfloat16) if bf16 else t

    def normal(self, shape, bf16=False, scale=1.0):
        h, t = self.empty(shape, bf16)
        t.normal_(0.0, scale, generator=self.gen)
        return h, t


def _positions(gen, B, seq):
    """Lengths spread over the last seven eighths of the cache, the longest sequence near its end."""
    pos = torch.randint(seq // 8, seq, (B,), generator=gen, device="cuda", dtype=torch.int32)
    pos[0] = seq - 1
    return pos


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def _prepare_attn(c, seed):
    m = _Memory(seed, c["asynchronous"])
    B, H, T, D, bf16 = c["B"], c["H"], c["T"], c["D"], c["dtype"] == "bf16"
    hc, ha = m.cuda.CreateCuDNN(), m.cuda.CreateAttn()
    m.cuda.SetAttn(hc, ha, 0, c["train"], B, T, H, D, 0.0, 0, ids.MCA_DTYPE_BF16 if bf16 else ids.MCA_DTYPE_F32,
                   ids.MCA_FLAG_CAUSAL_IMPLICIT if c["mask"] == "flag" else 0)
    s = dict(m=m, case=c, hc=hc, ha=ha, mask=0)
    if c["mask"] == "handle":
        s["mask"], t = m.empty((T, T))
        t.copy_(torch.tril(torch.ones(T, T, device="cuda")))
    elif c["mask"] == "key":       # padded sentences: each item has its own length
        s["mask"], t = m.empty((B, T))
        n = torch.randint(max(1, T // 2), T + 1, (B, 1), generator=m.gen, device="cuda")
        t.copy_((torch.arange(T, device="cuda")[None, :] < n).float())
    if c["packed"]:
        s["qkv"] = m.normal((B, T, 3 * H * D), bf16)
        s["y"] = m.empty((B, T, H * D), bf16)
        if c["train"]:
            s["dy"] = m.normal((B, T, H * D), bf16)
            s["dqkv"] = m.empty((B, T, 3 * H * D), bf16)
    else:
        shape = (B, H, T, D)
        s["q"], s["k"], s["v"] = (m.normal(shape, bf16) for _ in range(3))
        s["y"] = m.empty(shape, bf16)
        if c["train"]:
            s["dy"] = m.normal(shape, bf16)
            s["dq"], s["dk"], s["dv"] = (m.empty(shape, bf16) for _ in range(3))
    return s


def _prepare_decode(c, seed):
    m = _Memory(seed, c["asynchronous"])
    B, H, kv, hs, seq, bf16 = c["B"], c["H"], c["kv"], c["hs"], c["seq"], c["bf16"]
    s = dict(m=m, case=c, handle=m.cuda.CreateDecode(B, H, kv, hs, seq, bf16))
    s["q"], s["k"], s["v"] = m.normal((B, H * hs)), m.normal((B, kv * hs)), m.normal((B, kv * hs))
    s["kc"], s["vc"] = (m.normal((B, seq, kv * hs), bf16) for _ in range(2))
    s["pos"] = m.empty((B,))
    s["pos"][1].view(torch.int32).copy_(_positions(m.gen, B, seq))
    s["out"] = m.empty((B, H * hs))
    return s


def _llama_shapes(c):
    L, dim, kv_dim, hidden = c["layers"], c["heads"] * c["hs"], c.get("kv", c["heads"]) * c["hs"], c["hidden"]
    cfg = dict(dim=dim, hidden_dim=hidden, n_layers=L, n_heads=c["heads"], n_kv_heads=c.get("kv", c["heads"]), vocab_size=c["vocab"],
               seq_len=c["seq"])
    return cfg, {"wq": (L, dim, dim), "wk": (L, kv_dim, dim), "wv": (L, kv_dim, dim), "wo": (L, dim, dim), "w1": (L, hidden, dim),
                 "w2": (L, dim, hidden), "w3": (L, hidden, dim), "wcls": (c["vocab"], dim)}


_NAMES = ("token_embedding_table", "rms_att_weight", "rms_ffn_weight", "rms_final_weight", "wq", "wk", "wv", "wo", "w1", "w2", "w3",
          "wcls")


def _llama_weights(c, gen):
    """fp32 weights on the GPU, scaled so that the residual stream keeps its size."""
    cfg, shapes = _llama_shapes(c)
    w = {n: torch.empty(s, device="cuda").normal_(0.0, 0.7 / math.sqrt(s[-1]), generator=gen) for n, s in shapes.items()}
    w["token_embedding_table"] = torch.empty(c["vocab"], cfg["dim"], device="cuda").normal_(generator=gen)
    for n, s in (("rms_att_weight", (c["layers"], cfg["dim"])), ("rms_ffn_weight", (c["layers"], cfg["dim"])), ("rms_final_weight", (cfg["dim"],))):
        w[n] = torch.empty(s, device="cuda").normal_(1.0, 0.1, generator=gen)
    return cfg, w


def _prepare_token(c, seed):
    """A model loaded from host weights, as from a checkpoint, with a context already in its caches."""
    gen = torch.Generator("cuda").manual_seed(int(seed))
    cfg, w = _llama_weights(c, gen)
    model = llama2.TransformerGpu(0, batch=c["B"], weights_bf16=c["bf16"], cache_bf16=c["bf16"], use_graph=True)
    model.load_weights(cfg, {n: t.cpu().numpy() for n, t in w.items()})
    model.key_cache.normal_(generator=gen)
    model.value_cache.normal_(generator=gen)
    tokens = torch.randint(0, c["vocab"], (c["B"],), generator=gen, device="cuda").tolist()
    return dict(case=c, model=model, tokens=tokens, pos=_positions(gen, c["B"], c["seq"]).tolist())


def _prepare_step(c, seed):
    """Weights, caches and workspace that live in the host program's own device memory."""
    lib = _lib.load()
    gen = torch.Generator("cuda").manual_seed(int(seed))
    cfg, w = _llama_weights(c, gen)
    wdt = torch.bfloat16 if c["bf16"] else torch.float32
    w = {n: (t if n in _NAMES[:4] else t.to(wdt)).contiguous() for n, t in w.items()}
    B, S, L, kv_dim = c["B"], c["seq"], c["layers"], c["kv"] * c["hs"]
    s = dict(case=c, lib=lib, w=w)
    s["kc"], s["vc"] = (torch.empty(L, B, S, kv_dim, device="cuda", dtype=wdt).normal_(generator=gen) for _ in range(2))
    tables = [np.empty((S, c["hs"] // 2), np.float32) for _ in range(2)]
    fp = C.POINTER(C.c_float)
    lib.mca_rope_tables_host(S, c["hs"], 10000.0, *(t.ctypes.data_as(fp) for t in tables))
    s["fr"], s["fi"] = (torch.from_numpy(t).cuda() for t in tables)
    s["cfg"] = llama2.McaLlamaConfig(**cfg)
    s["weights"] = llama2.McaLlamaWeights(*[w[n].data_ptr() for n in _NAMES], int(c["bf16"]))
    n = lib.mca_llama_workspace_floats(C.byref(s["cfg"]), B, S)
    s["ws"] = torch.empty(n, device="cuda")
    s["st"] = llama2.McaLlamaState(s["kc"].data_ptr(), s["vc"].data_ptr(), int(c["bf16"]), s["fr"].data_ptr(), s["fi"].data_ptr(),
                                   s["ws"].data_ptr(), n)
    s["tokens"] = torch.randint(0, c["vocab"], (B,), generator=gen, device="cuda", dtype=torch.int32)
    s["pos"] = _positions(gen, B, S)
    s["logits"] = torch.empty(B, c["vocab"], device="cuda")
    return s


def _prepare_tft(c, seed):
    m = _Memory(seed, c["asynchronous"])
    B, H, Nq, Nk, d = c["B"], c["H"], c["Nq"], c["Nk"], c["d"]
    s = dict(m=m, case=c)
    s["q"], s["k"], s["v"] = m.normal((B, H, Nq, d)), m.normal((B, H, Nk, d)), m.normal((B, Nk, d))
    s["mask"] = m.empty((Nq, Nk))   # the query rows are the last Nq steps; later steps are masked (1)
    i, j = torch.arange(Nq, device="cuda")[:, None], torch.arange(Nk, device="cuda")[None, :]
    s["mask"][1].copy_((j > i + Nk - Nq).float())
    s["out"], s["attn"] = m.empty((B, Nq, d)), m.empty((B, Nq, Nk))
    s["dout"] = m.normal((B, Nq, d))
    s["dq"], s["dk"], s["dv"] = m.empty((B, H, Nq, d)), m.empty((B, H, Nk, d)), m.empty((B, Nk, d))
    return s


def _prepare_norm(c, seed):
    m = _Memory(seed, c["asynchronous"])
    shape = (c["rows"], c["inner"])
    s = dict(m=m, case=c, x=m.normal(shape), dy=m.normal(shape), y=m.empty(shape), dx=m.empty(shape))
    if c["op"] == "layernorm":
        s["handle"] = m.cuda.CreateLayerNorm(0, shape[0] * shape[1], 1, shape[0], shape[1], 1e-5)
    else:
        s["w"], s["inv"], s["dw"] = m.normal((shape[1],)), m.empty((shape[0],)), m.empty((shape[1],))
    return s


_PREPARE = {"attn": _prepare_attn, "decode": _prepare_decode, "token": _prepare_token, "step": _prepare_step, "tft": _prepare_tft,
            "norm": _prepare_norm}

# ------------------------------------------------------------------------------------------------------------- one pass


def run(state):
    return _RUN[state["case"]["kind"]](state)


def _run_attn(s):
    c, cuda = s["case"], s["m"].cuda
    key = c["mask"] == "key"
    if c["packed"]:
        cuda.AttnScaledDotProductForwardPacked(s["hc"], s["ha"], c["T"], s["qkv"][0], s["mask"], s["y"][0], key)
        if not c["train"]:
            return s["y"][1]
        cuda.AttnScaledDotProductBackwardPacked(s["hc"], s["ha"], s["qkv"][0], s["dqkv"][0], 0, s["y"][0], s["dy"][0])
        return s["y"][1], s["dqkv"][1]
    cuda.AttnScaledDotProductForward(s["hc"], s["ha"], c["T"], s["q"][0], s["k"][0], s["v"][0], s["mask"], s["y"][0], key)
    if not c["train"]:
        return s["y"][1]
    cuda.AttnScaledDotProductBackward(s["hc"], s["ha"], s["q"][0], s["dq"][0], s["k"][0], s["dk"][0], s["v"][0], s["dv"][0], 0,
                                      s["y"][0], s["dy"][0])
    return s["y"][1], s["dq"][1], s["dk"][1], s["dv"][1]


def _run_decode(s):
    s["m"].cuda.DecodeStep(s["handle"], s["q"][0], s["k"][0], s["v"][0], s["kc"][0], s["vc"][0], s["pos"][0], s["case"]["seq"], s["out"][0])
    return s["out"][1], s["kc"][1], s["vc"][1]


def _run_token(s):
    model = s["model"]
    logits = model.forward(s["tokens"][0], s["pos"][0]) if s["case"]["B"] == 1 else model.forward_batch(s["tokens"], s["pos"])
    return logits, model.key_cache, model.value_cache


def _run_step(s):
    rc = s["lib"].mca_llama_forward(C.byref(s["cfg"]), C.byref(s["weights"]), C.byref(s["st"]), s["tokens"].data_ptr(), s["pos"].data_ptr(),
                                    s["case"]["B"], s["case"]["seq"], s["logits"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    if rc:
        raise RuntimeError(f"mca_llama_forward failed with {rc}")
    return s["logits"], s["kc"], s["vc"]


def _run_tft(s):
    c, cuda = s["case"], s["m"].cuda
    sizes = (c["B"], c["H"], c["Nq"], c["Nk"], c["d"])
    cuda.TftAttnForward(s["q"][0], s["k"][0], s["v"][0], s["mask"][0], *sizes, s["out"][0], s["attn"][0])
    cuda.TftAttnBackward(s["q"][0], s["k"][0], s["v"][0], s["mask"][0], s["dout"][0], 0, *sizes, s["dq"][0], s["dk"][0], s["dv"][0])
    return [s[n][1] for n in ("out", "attn", "dq", "dk", "dv")]


def _run_norm(s):
    c, cuda = s["case"], s["m"].cuda
    if c["op"] == "layernorm":
        cuda.LayerNormForward(s["handle"], s["x"][0], s["y"][0])
        cuda.LayerNormBackward(s["handle"], s["y"][0], s["dy"][0], s["dx"][0])
        return s["y"][1], s["dx"][1]
    cuda.RmsNormForward(s["x"][0], s["w"][0], s["y"][0], s["inv"][0], c["rows"], c["inner"])
    cuda.RmsNormBackward(s["x"][0], s["w"][0], s["dy"][0], s["inv"][0], s["dx"][0], s["dw"][0], c["rows"], c["inner"])
    return s["y"][1], s["dx"][1], s["dw"][1]


_RUN = {"attn": _run_attn, "decode": _run_decode, "token": _run_token, "step": _run_step, "tft": _run_tft, "norm": _run_norm}

# ----------------------------------------------------------------------------------------------------- work, tolerances


def work(c):
    """Inputs once, outputs once, and the products of the algorithm: two contractions forward, five backward (the
    scores again); causal ones over the lower triangle.  Decode: mean length 9/16 of the cache."""
    if c["kind"] == "attn":
        B, H, T, D = c["B"], c["H"], c["T"], c["D"]
        n, size = B * H * T * D, 2 if c["dtype"] == "bf16" else 4
        pairs = B * H * (T * T if c["mask"] == "key" else T * (T + 1) / 2)
        mask = 4 * {"handle": T * T, "key": B * T, "flag": 0}[c["mask"]]
        return {"bytes": n * size * (4 + (7 if c["train"] else 0)) + mask, "flops": pairs * D * (4 + (10 if c["train"] else 0))}
    if c["kind"] == "decode":
        size, rows = 2 if c["bf16"] else 4, c["B"] * c["seq"] * 9 / 16
        return {"bytes": 2 * rows * c["kv"] * c["hs"] * size + 8 * c["B"] * c["H"] * c["hs"], "flops": 4 * rows * c["H"] * c["hs"]}
    if c["kind"] in ("token", "step"):
        cfg, shapes = _llama_shapes(c)
        size, weights = 2 if c["bf16"] else 4, sum(int(np.prod(s)) for s in shapes.values())
        rows = c["B"] * c["seq"] * (1.0 if c["B"] == 1 else 9 / 16) * c["layers"]
        return {"bytes": (weights + 2 * rows * cfg["n_kv_heads"] * c["hs"]) * size + 4 * c["B"] * c["vocab"],
                "flops": 2 * c["B"] * weights + 4 * rows * cfg["dim"]}
    if c["kind"] == "tft":
        B, H, Nq, Nk, d = c["B"], c["H"], c["Nq"], c["Nk"], c["d"]
        heads, shared, rows = B * H * (Nq + Nk) * d, B * Nk * d, B * Nq * d
        return {"bytes": 4 * (heads + shared + Nq * Nk + rows + B * Nq * Nk + 2 * heads + 2 * shared + rows + Nq * Nk),
                "flops": B * Nq * Nk * d * (2 * H + 2 + 6 * H + 4)}
    return {"bytes": 4 * c["rows"] * c["inner"] * 5, "flops": 16 * c["rows"] * c["inner"]}


def tolerance(c):
    """bf16 tensors or weights: bf16's rounding.  fp32: sums of fp32 products in another order."""
    if c.get("dtype") == "bf16" or (c["kind"] in ("token", "step") and c["bf16"]):
        return {"rel": 1e-2}
    return {"rel": 2e-5}
