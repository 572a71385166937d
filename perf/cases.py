"""The work a user has this library do, as timed cases.

Every case goes through the public operators: `lightning_attn_func` (scalar and vector decay, forward
only or forward and backward, batched or packed with `cu_seqlens`), the single-token decode steps, and
a gated block's attention followed by `normalize_gate_fn`.  Sizes are those of the benchmark
configurations and of the tests, plus generic ones between them.

A case is a dict of plain values:
  op      "decode" | "attn" | "block"
  decay   "scalar" | "vector"
  B, N, H, D   batch, tokens per sequence (packed: of the whole stream), heads, features per head
  docs    0, or the number of documents of a packed stream (B = 1 then)
  train   False: forward only (no_grad); True: forward and backward, all gradients returned
  gates   scalar decay: "head" = a constant per head, "token" = logsigmoid of a projection per token;
          vector decay: "mild" = logsigmoid(x)/16 in fp32, "full" = logsigmoid(x) in the 16-bit type
  state   whether an initial state is given (decode always carries one)
  dtype   type of q, k, v
"""
import math

import torch
import torch.nn.functional as F

from xopes_b200 import lasd_decode_step, lavd_decode_step, lightning_attn_func
from xopes_b200.normalize import normalize_gate_fn

_DTYPES = {"bfloat16": torch.bfloat16, "float16": torch.float16, "float32": torch.float32}


def _case(name=None, *, op="attn", decay="scalar", B=1, N=1, H=16, D=128, docs=0, train=False, gates="head",
          state=False, dtype="bfloat16"):
    c = dict(op=op, decay=decay, B=B, N=N, H=H, D=D, docs=docs, train=train, gates=gates, state=state, dtype=dtype)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # one user's stream, one layer's token: latency of a single call
        _case("decode_scalar_b1", op="decode", B=1, H=16),
        # a serving batch in mid-size with per-feature decays
        _case("decode_vector_b32", op="decode", decay="vector", gates="mild", B=32, H=32),
        # the benchmark's decode batch: the state is streamed from HBM and back
        _case("decode_scalar_b256", op="decode", B=256, H=32),
        # the benchmark's fp32 forward: evaluation and checks in full precision
        _case("fwd_fp32_b2_n512", B=2, N=512, H=8, D=64, dtype="float32"),
        # prefill of one prompt of a ragged length, the state kept for decoding
        _case("prefill_b1_n1000", B=1, N=1000, H=32, state=True),
        # the benchmark's training step: large batch, a constant decay per head
        _case("train_scalar_b8_n8192", B=8, N=8192, H=32, train=True, state=True),
        # a gated block as the training tests shape it: per-token decays with their gradient, narrow
        # heads, the normalisation and gate behind the attention
        _case("block_b8_n2048_d64", op="block", B=8, N=2048, H=12, D=64, train=True, gates="token"),
        # one long document: few pairs of sequence and head, each very long
        _case("train_scalar_b1_n32768", B=1, N=32768, H=16, train=True),
        # the benchmark's packed stream: a million tokens in ragged documents, forward
        _case("packed_fwd_1m", N=1 << 20, H=16, docs=64),
        # packed training batch of ragged documents with per-token decays
        _case("packed_train_32k", N=32768, H=16, docs=24, train=True, gates="token"),
        # the benchmark's vector-decay training step
        _case("train_vector_b4_n16384", decay="vector", B=4, N=16384, H=16, train=True, gates="mild"),
        # vector decay as the upstream benchmark draws it: unscaled logsigmoid in the 16-bit type
        _case("train_vector_full_n4096", decay="vector", B=2, N=4096, H=16, train=True, gates="full"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: the same kinds of call, sizes spread over their range, most of them odd."""
    kind = rng.choice(["decode", "decode", "fwd_fp32", "prefill", "prefill", "train_scalar", "train_scalar",
                       "train_token", "block", "packed_fwd", "packed_train", "train_vector", "train_vector",
                       "train_vector_full"])
    dtype = rng.choice(["bfloat16", "bfloat16", "bfloat16", "float16"])
    if kind == "decode":
        vector = rng.random() < 0.5
        return _case(op="decode", decay="vector" if vector else "scalar", gates="mild" if vector else "head",
                     B=_log_int(rng, 1, 256), H=rng.choice([8, 12, 16, 32]), D=rng.choice([64, 128, 128]), dtype=dtype)
    if kind == "fwd_fp32":
        return _case(B=rng.choice([1, 2, 3]), N=_log_int(rng, 100, 2048), H=rng.choice([4, 8, 12]),
                     D=rng.choice([32, 64, 128]), dtype="float32", state=rng.random() < 0.5)
    if kind == "prefill":
        return _case(B=rng.choice([1, 1, 2, 4]), N=_log_int(rng, 60, 8192), H=rng.choice([16, 32]),
                     D=rng.choice([64, 128, 128]), state=rng.random() < 0.5, gates=rng.choice(["head", "token"]),
                     dtype=dtype)
    if kind in ("train_scalar", "train_token"):
        n = _log_int(rng, 400, 32768)
        h = rng.choice([12, 16, 32])
        b = rng.randint(1, max(1, min(8, (8 * 8192 * 32) // (n * h))))
        return _case(B=b, N=n, H=h, D=rng.choice([64, 128, 128]), train=True, state=rng.random() < 0.5,
                     gates="head" if kind == "train_scalar" else "token", dtype=dtype)
    if kind == "block":
        return _case(op="block", B=rng.randint(1, 8), N=_log_int(rng, 500, 4096), H=rng.choice([8, 12, 16]),
                     D=rng.choice([64, 128]), train=True, gates="token", dtype=dtype)
    if kind == "packed_fwd":
        n = _log_int(rng, 8000, 1 << 19)
        return _case(N=n, H=16, docs=rng.randint(2, 64), dtype=dtype, gates=rng.choice(["head", "token"]))
    if kind == "packed_train":
        return _case(N=_log_int(rng, 4000, 131072), H=rng.choice([8, 16]), docs=rng.randint(2, 48), train=True,
                     gates="token", dtype=dtype)
    n = _log_int(rng, 500, 16384)
    return _case(decay="vector", B=rng.randint(1, max(1, min(4, 65536 // n))), N=n, H=rng.choice([8, 16]), train=True,
                 gates="full" if kind == "train_vector_full" else "mild", state=rng.random() < 0.3, dtype="bfloat16")


def _randn(gen, shape, dtype=torch.float32, scale=1.0):
    # in blocks along the tokens so that the fp32 draw of a long stream stays small
    if len(shape) == 4 and shape[0] * shape[1] > 65536:
        out = torch.empty(shape, dtype=dtype, device="cuda")
        flat = out.view(-1, *shape[2:])
        for a in range(0, flat.shape[0], 65536):
            part = flat[a:a + 65536]
            part.copy_(torch.randn(part.shape, generator=gen, device="cuda").mul_(scale))
        return out
    return torch.randn(shape, generator=gen, device="cuda").mul_(scale).to(dtype)


def _head_decay(h, step):
    """log(1 - 2^(-5 - step * i)) for head i."""
    return torch.log(1 - torch.pow(2.0, -5 - step * torch.arange(h, dtype=torch.float32))).cuda()


def _boundaries(gen, n, docs):
    """Uniform-random document lengths normalised to the stream, at least one token each."""
    w = torch.rand(docs, generator=gen, device="cuda")
    lens = torch.floor(w / w.sum() * (n - docs)).to(torch.int64) + 1
    lens[-1] += n - lens.sum()
    cu = torch.zeros(docs + 1, dtype=torch.int64, device="cuda")
    cu[1:] = torch.cumsum(lens, 0)
    return cu


def prepare(case, seed):
    b, n, h, d = case["B"], case["N"], case["H"], case["D"]
    dtype = _DTYPES[case["dtype"]]
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 13)
    train = case["train"]
    s = {"case": case}
    if case["op"] == "decode":
        for x in "qkv":
            s[x] = _randn(gen, (b, 1, h, d), dtype, d ** -0.5)
        s["state"] = _randn(gen, (b, h, d, d), torch.float32, 0.1)
        if case["decay"] == "vector":
            s["ldk"] = F.logsigmoid(_randn(gen, (b, 1, h, d))) / 16
        else:
            s["ld"] = _head_decay(h, 8.0 / h)
        return s
    vector = case["decay"] == "vector"
    s["v"] = _randn(gen, (b, n, h, d), dtype)
    if vector:
        x = _randn(gen, (b, n, h, d))
        ldk = F.logsigmoid(x)
        if case["gates"] == "mild":
            ldk = ldk / 16
            s["k"] = ((1 - torch.exp(ldk)) * _randn(gen, (b, n, h, d), torch.float32, d ** -0.5)).to(dtype)
            s["q"] = _randn(gen, (b, n, h, d), dtype)
        else:
            ldk = ldk.to(dtype)
            s["k"] = _randn(gen, (b, n, h, d), dtype, d ** -0.5)
            s["q"] = _randn(gen, (b, n, h, d), dtype, d ** -0.5)
        s["ldk"] = ldk
    else:
        s["q"] = _randn(gen, (b, n, h, d), dtype, d ** -0.5)
        s["k"] = _randn(gen, (b, n, h, d), dtype, d ** -0.5)
        if case["gates"] == "head":
            s["ld"] = _head_decay(h, 8.0 / h)
        else:
            s["ld"] = F.logsigmoid(_randn(gen, (b, n, h)) + 2.0)
    s["cu"] = _boundaries(gen, n, case["docs"]) if case["docs"] else None
    s["s0"] = _randn(gen, (case["docs"] or b, h, d, d), torch.float32, 0.1) if case["state"] else None
    if case["op"] == "block":
        s["gate"] = _randn(gen, (b, n, h * d), dtype)
        s["weight"] = (1.0 + 0.1 * _randn(gen, (h * d,))).to(dtype)
    if train:
        s["do"] = _randn(gen, (b, n, h * d) if case["op"] == "block" else (b, n, h, d), dtype)
        wanted = ["q", "k", "v"]
        if vector:
            wanted.append("ldk")
        elif case["gates"] == "token":
            wanted.append("ld")
        if case["op"] == "block":
            wanted += ["gate", "weight"]
        for x in wanted:
            s[x].requires_grad_()
        s["wanted"] = wanted
    return s


def _attend(s):
    return lightning_attn_func(s["q"], s["k"], s["v"], ld=s.get("ld"), ldk=s.get("ldk"), initial_state=s["s0"],
                               cu_seqlens=s["cu"], decay_type=s["case"]["decay"])


def run(s):
    case = s["case"]
    if case["op"] == "decode":
        if case["decay"] == "vector":
            return lavd_decode_step(s["q"], s["k"], s["v"], s["ldk"], s["state"])
        return lasd_decode_step(s["q"], s["k"], s["v"], s["ld"], s["state"])
    if not case["train"]:
        with torch.no_grad():
            return _attend(s)
    o, state = _attend(s)
    if case["op"] == "block":
        o = normalize_gate_fn(o.reshape(case["B"], case["N"], -1), s["weight"], gate=s["gate"], gate_act="sigmoid",
                              gate_pos="pre", c=case["D"] ** 0.5, num_groups=case["H"])
    grads = torch.autograd.grad(o, [s[x] for x in s["wanted"]], s["do"])
    return (o.detach(), state.detach()) + grads


def work(case):
    """Inputs once, outputs once; operations of the recurrence itself (state update and read-out
    forward; states again, their gradient and three read-outs backward)."""
    b, n, h, d = case["B"], case["N"], case["H"], case["D"]
    size = 4 if case["dtype"] == "float32" else 2
    th = b * n * h                      # token-heads
    states = (case["docs"] or b) * h * d * d * 4
    if case["op"] == "decode":
        decay = th * d * 4 if case["decay"] == "vector" else h * 4
        return {"bytes": 4 * th * d * size + 2 * states + decay, "flops": 6 * th * d * d}
    if case["decay"] == "vector":
        decay = th * d * (4 if case["gates"] == "mild" else size)
    else:
        decay = h * 4 if case["gates"] == "head" else th * 4
    rows = 8 if case["train"] else 4    # q k v o, and do dq dk dv
    if case["op"] == "block":
        rows += 2                       # gate and its gradient
    decays = 1 if not case["train"] or (case["decay"] == "scalar" and case["gates"] == "head") else 2
    total = rows * th * d * size + decays * decay + (2 if case["state"] else 1) * states
    return {"bytes": total, "flops": (14 if case["train"] else 4) * th * d * d}


def tolerance(case):
    """About four times the measured difference between the result and the recurrence in 64 bits
    (largest of all outputs; rel, max): bf16 3.3e-3, 4e-2 (a block's decay gradient 4.2e-3), fp16
    3.4e-4, 2.4e-3, fp32 6e-7, 6e-6.  A decode step's sums are all fp32 (its state 4e-8) and only
    its output is rounded, where a tie may fall the other way."""
    if case["op"] == "decode":
        return {"rel": 3e-4, "max": 1e-3} if case["dtype"] == "float16" else {"rel": 2e-3, "max": 8e-3}
    if case["dtype"] == "float32":
        return {"rel": 2.4e-6, "max": 2.4e-5}
    if case["dtype"] == "float16":
        return {"rel": 1.4e-3, "max": 1e-2}
    return {"rel": 1.3e-2, "max": 0.16}
