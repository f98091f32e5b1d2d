"""The work that a user of this package has it do, as cases that can be timed.

A case names one of eight paths through the public entry points and its sizes:

* ``train``: ``AttentionEngine(...)(q, k, v)`` under autograd and its backward; softmax, sigmoid or ReLU scores; causal,
  full, sliding-window or call-time block masks; MHA and GQA; fp16 and bf16; head dims 64 and 128
* ``prefill``: the same call without gradients
* ``decode``: a decode engine (``q_len != kv_len``) on a batch whose rows have the same length
* ``decode_rows``: ``decode_varlen`` on rows of different lengths, dense or paged, under a schedule made once per step
* ``mla``: the kv-shared (MLA) decode ``engine(q, q_pe, kv, k_pe)``
* ``mla_paged``: ``decode_paged`` over a pool of 64-key pages, one length per row
* ``scan_train``: ``LinearAttentionEngine`` under autograd and its backward: the Mamba2 block with its skip connection, or
  gated linear attention (``q_mod`` and a log-decay)
* ``scan``: the same call without gradients

Engines are kept per problem, as a program keeps them; inputs are made on the GPU from the seed.
"""
import functools
import math

import torch

from attentionengine_b200 import AttentionEngine, CustomIO, LinearAttentionEngine, examples, meta_tensor

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
_DEV = "cuda"


def listed():
    return [
        # one small training step: four heads of 64 over 512 positions, where launches and host work are what counts
        dict(name="train_mha_512", path="train", score="softmax", mask="causal", B=1, Hq=4, Hkv=4, S=512, D=64,
             dtype="fp16"),
        # the attention of one Llama-3.1-8B layer in training at 8K context
        dict(name="train_gqa_8k", path="train", score="softmax", mask="causal", B=8, Hq=32, Hkv=8, S=8192, D=128,
             dtype="fp16"),
        # a local-attention layer on sequences that do not fill their last tile
        dict(name="train_window_4000", path="train", score="softmax", mask="window", window=1024, B=2, Hq=16, Hkv=4,
             S=4000, D=128, dtype="bf16"),
        # sigmoid attention in training: no row statistics, every tile visited
        dict(name="train_sigmoid_4k", path="train", score="sigmoid", mask="full", B=4, Hq=32, Hkv=32, S=4096, D=128,
             dtype="bf16"),
        # one prompt of an odd length before decoding starts
        dict(name="prefill_gqa_3001", path="prefill", score="softmax", mask="causal", B=1, Hq=32, Hkv=8, S=3001, D=128,
             dtype="bf16"),
        # a short chat: two rows, one thousand cached keys, one new position
        dict(name="decode_gqa_2x1000", path="decode", B=2, Hq=32, Hkv=8, Sq=1, Skv=1000, D=128, dtype="fp16"),
        # a decode step of a full batch at 8K context
        dict(name="decode_gqa_16x8k", path="decode", B=16, Hq=32, Hkv=8, Sq=1, Skv=8192, D=128, dtype="fp16"),
        # continuous batching: 64 rows of lengths from 1 to 8192 over a paged cache
        dict(name="decode_paged_64", path="decode_rows", paged=True, B=64, Hq=32, Hkv=8, Skv=8192, D=128, dtype="bf16"),
        # DeepSeek-V3 decode, a full batch at 8K context
        dict(name="mla_128x8k", path="mla", B=128, H=128, S=8192, dtype="fp16"),
        # DeepSeek-V3 decode from a paged cache, a few rows of different lengths
        dict(name="mla_paged_8x4k", path="mla_paged", B=8, H=128, S=4096, dtype="bf16"),
        # the Mamba2 block in training: 80 heads of 64, state 128, 8K steps
        dict(name="scan_train_8k", path="scan_train", kind="mamba2", B=8, H=80, T=8192, DK=128, DV=64, dtype="bf16"),
        # the Mamba2 block over one short prompt
        dict(name="scan_1000", path="scan", kind="mamba2", B=1, H=80, T=1000, DK=128, DV=64, dtype="bf16"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


_MOST_TRAIN = 3.5 * 4.0 * 8 * 32 * 8192 * 8192 * 128 / 2


def draw(rng):
    path = rng.choice(["train", "train", "prefill", "decode", "decode_rows", "mla", "mla_paged", "scan_train", "scan"])
    dtype = rng.choice(["fp16", "bf16"])
    if path in ("train", "prefill"):
        score = rng.choice(["softmax", "softmax", "softmax", "sigmoid", "relu"])
        mask = rng.choice(["causal", "causal", "full", "window", "blocks"]) if score == "softmax" else rng.choice(["causal", "full"])
        while True:
            Hkv = rng.choice([1, 2, 4, 8])
            Hq = Hkv * (rng.choice([1, 1, 4, 8]) if score == "softmax" else 1)
            c = dict(path=path, score=score, mask=mask, B=_log_int(rng, 1, 8), Hq=Hq, Hkv=Hkv, S=_log_int(rng, 128, 8192),
                     D=rng.choice([64, 128, 128]), dtype=dtype)
            if mask == "window":
                c["window"] = _log_int(rng, 64, 4096)
            if work(c)["flops"] <= _MOST_TRAIN:
                return c
    if path in ("decode", "decode_rows"):
        Hkv = rng.choice([4, 8, 32])
        c = dict(path=path, B=_log_int(rng, 1, 64), Hq=32, Hkv=Hkv, Skv=_log_int(rng, 128, 16384 if Hkv < 32 else 4096),
                 D=rng.choice([64, 128, 128]), dtype=dtype)
        c.update({"Sq": 1} if path == "decode" else {"paged": rng.choice([True, False])})
        return c
    if path == "mla":
        return dict(path=path, B=_log_int(rng, 1, 128), H=rng.choice([16, 64, 128, 128]), S=_log_int(rng, 128, 8192), dtype=dtype)
    if path == "mla_paged":
        return dict(path=path, B=_log_int(rng, 1, 64), H=rng.choice([16, 64, 128, 128]), S=_log_int(rng, 256, 8192), dtype=dtype)
    if rng.random() < 0.7:
        return dict(path=path, kind="mamba2", B=_log_int(rng, 1, 8), H=rng.choice([8, 24, 48, 80]), T=_log_int(rng, 128, 8192),
                    DK=128, DV=64, dtype=dtype)
    return dict(path=path, kind="gla", B=_log_int(rng, 1, 4), H=rng.choice([4, 8, 16]), T=_log_int(rng, 128, 4096),
                DK=rng.choice([128, 256]), DV=rng.choice([64, 128, 256]), dtype=dtype)


# ---------------------------------------------------------------------------------------------------- engines
@functools.lru_cache(maxsize=None)
def _attention(score, mask, window, B, Hq, Hkv, S, D, dtype):
    dt, scale = _DTYPES[dtype], 1.0 / math.sqrt(D)
    causal = mask == "causal"
    if score == "sigmoid":
        return examples.sigmoid_engine(B, Hq, S, D, dt, causal)
    if score == "relu":
        return examples.relu_engine(B, Hq, S, D, dt, causal, post_scale=1.0 / S)
    if mask in ("causal", "full"):
        return examples.softmax_engine(B, Hq, Hkv, S, D, D, dt, causal)

    def score_mod(s, custom, b, h, q_idx, kv_idx):
        return s * scale

    def window_mask(b, h, q_idx, kv_idx):
        return torch.logical_and(q_idx >= kv_idx, q_idx - kv_idx <= window)

    return AttentionEngine(examples.metas(B, Hq, Hkv, S, D, D, dt), CustomIO({}), score_mod=score_mod,
                           mask_mod=window_mask if mask == "window" else None, online_func=examples.OnlineSoftmax(),
                           extern_block_mask=mask == "blocks")


@functools.lru_cache(maxsize=None)
def _decode(B, Hq, Hkv, Sq, Skv, D, dtype):
    return examples.decode_engine(B, Hq, Hkv, Sq, Skv, D, _DTYPES[dtype])


@functools.lru_cache(maxsize=None)
def _mla(B, H, S, dtype):
    return examples.mla_engine(B, H, S, _DTYPES[dtype], 1.0 / math.sqrt(192))


@functools.lru_cache(maxsize=None)
def _linear(kind, B, H, T, DK, DV, dtype):
    dt = _DTYPES[dtype]
    if kind == "mamba2":
        return examples.mamba2_engine(B, H, T, DK, DV, dt, d_skip=True)
    scale = 1.0 / math.sqrt(DK)
    metas = tuple(meta_tensor(B, H, T, n, dtype=dt) for n in (DK, DK, DV))
    return LinearAttentionEngine(metas, q_mod=lambda q, io: q * scale, custom_io=CustomIO({}))


# ---------------------------------------------------------------------------------------------------- inputs
def _lengths(B, longest, gen):
    """One length per row, uniform from 1 to ``longest``; the first row has the longest."""
    n = torch.randint(1, longest + 1, (B,), generator=gen, device=_DEV, dtype=torch.int32)
    n[0] = longest
    return n


def prepare(case, seed):
    c = case
    gen = torch.Generator(device=_DEV).manual_seed(seed)
    dt = _DTYPES[c["dtype"]]

    def normal(*shape, dtype=dt):
        return torch.randn(*shape, generator=gen, device=_DEV, dtype=dtype)

    s = {"path": c["path"]}
    if c["path"] in ("train", "prefill"):
        B, Hq, Hkv, S, D = (c[n] for n in ("B", "Hq", "Hkv", "S", "D"))
        s["engine"] = _attention(c["score"], c["mask"], c.get("window", 0), B, Hq, Hkv, S, D, c["dtype"])
        s["qkv"] = [normal(B, S, Hq, D), normal(B, S, Hkv, D), normal(B, S, Hkv, D)]
        s["custom"] = [torch.tensor([-math.log(S)], device=_DEV)] if c["score"] == "sigmoid" else []
        s["keywords"] = {}
        if c["mask"] == "blocks":  # half of the blocks, the diagonal always
            n = -(-S // 128)
            blocks = torch.rand(1, Hq, n, n, generator=gen, device=_DEV) < 0.5
            s["keywords"] = {"block_mask": (blocks | torch.eye(n, device=_DEV, dtype=torch.bool)).to(torch.int8)}
        if c["path"] == "train":
            s["d_o"] = normal(B, S, Hq, D)
            for t in s["qkv"]:
                t.requires_grad_()
    elif c["path"] == "decode":
        s["engine"] = _decode(c["B"], c["Hq"], c["Hkv"], c["Sq"], c["Skv"], c["D"], c["dtype"])
        s["qkv"] = [normal(c["B"], c["Sq"], c["Hq"], c["D"]), normal(c["B"], c["Skv"], c["Hkv"], c["D"]),
                    normal(c["B"], c["Skv"], c["Hkv"], c["D"])]
    elif c["path"] == "decode_rows":
        B, Skv = c["B"], c["Skv"]
        s["engine"] = _decode(B, c["Hq"], c["Hkv"], 1, Skv, c["D"], c["dtype"])
        s["lengths"] = _lengths(B, Skv, gen)
        s["schedule"] = s["engine"].decode_schedule(s["lengths"])  # once per step, for all layers of a model
        q = normal(B, 1, c["Hq"], c["D"])
        if c["paged"]:
            pages = -(-Skv // 128)
            s["table"] = torch.randperm(B * pages, generator=gen, device=_DEV).to(torch.int32).view(B, pages)
            s["qkv"] = [q, normal(B * pages, 128, c["Hkv"], c["D"]), normal(B * pages, 128, c["Hkv"], c["D"])]
        else:
            s["table"] = None
            s["qkv"] = [q, normal(B, Skv, c["Hkv"], c["D"]), normal(B, Skv, c["Hkv"], c["D"])]
    elif c["path"] == "mla":
        B, H, S = c["B"], c["H"], c["S"]
        s["engine"] = _mla(B, H, S, c["dtype"])
        s["args"] = [normal(B, 1, H, 512), normal(B, 1, H, 64), normal(B, S, 1, 512), normal(B, S, 1, 64)]
    elif c["path"] == "mla_paged":
        B, H, S = c["B"], c["H"], c["S"]
        s["engine"] = _mla(B, H, S, c["dtype"])
        pages = -(-S // 64)
        s["args"] = [normal(B, 1, H, 576), normal(B * pages, 64, 1, 576),
                     torch.randperm(B * pages, generator=gen, device=_DEV).to(torch.int32).view(B, pages),
                     _lengths(B, S, gen)]
    else:
        B, H, T, DK, DV = (c[n] for n in ("B", "H", "T", "DK", "DV"))
        s["engine"] = _linear(c["kind"], B, H, T, DK, DV, c["dtype"])
        if c["kind"] == "mamba2":
            x, Bm, Cm = normal(B, H, T, DV), normal(B, 1, T, DK), normal(B, 1, T, DK)
            step = torch.nn.functional.softplus(normal(B, H, T, dtype=torch.float32) - 4.0)
            A = -torch.exp(torch.rand(1, H, generator=gen, device=_DEV) * math.log(16.0))
            s["args"] = [Cm, Bm, x, step, A, step.to(dt), normal(1, H, dtype=torch.float32)]
        else:
            decay = torch.nn.functional.logsigmoid(normal(B, H, T, dtype=torch.float32)) / 16
            s["args"] = [normal(B, H, T, DK), normal(B, H, T, DK), normal(B, H, T, DV), decay]
        if c["path"] == "scan_train":
            s["d_o"] = normal(B, H, T, DV)
            for t in s["args"]:
                t.requires_grad_()
    return s


def run(state):
    s = state
    path, engine = s["path"], s["engine"]
    if path in ("train", "scan_train"):
        leaves = s["qkv"] if path == "train" else s["args"]
        for t in leaves:
            t.grad = None
        o = engine(*leaves, *s["custom"], **s["keywords"]) if path == "train" else engine(*leaves)
        o.backward(s["d_o"])
        return [o.detach()] + [t.grad for t in leaves]
    if path == "prefill":
        with torch.no_grad():
            return engine(*s["qkv"], *s["custom"], **s["keywords"])
    if path == "decode":
        return engine(*s["qkv"])
    if path == "decode_rows":
        return engine.decode_varlen(*s["qkv"], s["lengths"], block_table=s["table"], metadata=s["schedule"])
    if path == "mla":
        return engine(*s["args"])
    if path == "mla_paged":
        return engine.decode_paged(*s["args"])
    with torch.no_grad():
        return engine(*s["args"])


# ---------------------------------------------------------------------------------------------------- what a pass needs
def _kept(c):
    """Expected number of (query, key) pairs of one head."""
    S = c["S"]
    if c["mask"] == "causal":
        return S * (S + 1) / 2
    if c["mask"] == "window":
        w = min(S, c["window"] + 1)
        return w * (w + 1) / 2 + (S - w) * w
    if c["mask"] == "blocks":
        n = -(-S // 128)
        return S * S * (0.5 + 0.5 / n)
    return float(S) * S


def work(case):
    c = case
    path = c["path"]
    if path in ("train", "prefill"):
        q, kv = c["B"] * c["S"] * c["Hq"] * c["D"], c["B"] * c["S"] * c["Hkv"] * c["D"]
        forward = 4.0 * c["B"] * c["Hq"] * _kept(c) * c["D"]
        if path == "prefill":
            return {"bytes": 2.0 * (2 * q + 2 * kv), "flops": forward}
        return {"bytes": 2.0 * (4 * q + 4 * kv), "flops": 3.5 * forward}
    if path in ("decode", "decode_rows"):
        # rows of different lengths: the first has Skv keys, the others (Skv + 1) / 2 on average
        keys = c["B"] * c["Skv"] if path == "decode" else c["Skv"] + (c["B"] - 1) * (c["Skv"] + 1) / 2
        return {"bytes": 2.0 * (2 * keys * c["Hkv"] * c["D"] + 2 * c["B"] * c["Hq"] * c["D"]), "flops": 4.0 * keys * c["Hq"] * c["D"]}
    if path in ("mla", "mla_paged"):
        keys = c["B"] * c["S"] if path == "mla" else c["S"] + (c["B"] - 1) * (c["S"] + 1) / 2
        return {"bytes": 2.0 * (keys * 576 + c["B"] * c["H"] * (576 + 512)), "flops": 2.0 * keys * c["H"] * (576 + 512)}
    B, H, T, DK, DV = (c[n] for n in ("B", "H", "T", "DK", "DV"))
    heads = 1 if c["kind"] == "mamba2" else H  # heads of q and k
    qk, v, rows = 2 * B * heads * T * DK, B * H * T * DV, 4.0 * B * H * T
    # chunks of 128 steps: q k^T per q / k head; per value head P v over the lower triangle, q h and k^T v
    forward = B * T * (heads * 128.0 * DK + H * 128.0 * DV + H * 4.0 * DK * DV)
    if path == "scan":
        return {"bytes": 2.0 * (qk + 2 * v) + rows, "flops": forward}
    return {"bytes": 2.0 * (2 * qk + 4 * v) + 2 * rows, "flops": 3.5 * forward}


def tolerance(case):
    # Scan in training: the gradient of a log-decay is a sum of many 16-bit products that nearly cancel, so it carries
    # about 1 % in bf16 and an eighth of that in fp16.  Everything else: operands rounded to 16 bits once or twice before a product.
    if case["path"] == "scan_train":
        return {"rel": 2e-2} if case["dtype"] == "bf16" else {"rel": 5e-3}
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 2e-3}
