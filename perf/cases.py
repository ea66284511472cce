"""The work that this framework's users have it do, as cases that can be timed and compared.

Two levels of entry point are used, as in users' programs: the `Castle` module (projections included: training
steps, prompts, token-by-token sampling) and the operators `castle_attention`, `castle_attention_packed` and
`castle_decode_step` (callers with projections or caches of their own).  A case's "kind" says which:

    module_decode   `tokens` cached single-token steps of a `Castle` module, one after the other
    module_prefill  a prompt through `Castle(..., return_next_cache=True)`: the output and the four caches
    module_train    a `Castle` module's forward and backward: the output and every gradient
    op_decode       `castle_decode_step` on four caches of the caller's
    op_forward      `castle_attention` on six (B, H, N, d) tensors, no gradients (scoring, evaluation)
    op_train        `castle_attention`, forward and backward: the output and six gradients
    packed_train    `castle_attention_packed` on the projection output (B, N, 6, H, d), forward and backward

"n" is the number of positions: of the sequence, or already in the caches where single tokens are decoded.
"""
import math

import torch

from lookahead_keys_attention_b200 import (Castle, cache_from_buffers, castle_attention, castle_attention_packed,
                                           castle_decode_step)

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _case(name, kind, dtype, batch, heads, dim_head, n, dim=0, tokens=1, prenorm=False, rotary=False):
    c = {"kind": kind, "dtype": dtype, "batch": batch, "heads": heads, "dim_head": dim_head, "n": n, "dim": dim,
         "tokens": tokens, "prenorm": prenorm, "rotary": rotary}
    return c if name is None else {"name": name, **c}


def listed():
    return [
        # The README's module and shape: fp32, two sequences of 128, continued token by token.
        _case("decode_readme_fp32", "module_decode", "fp32", 2, 8, 64, 128, dim=512, tokens=8),
        # Sampling from one layer of the byte language model, which has pre-norm and rotary: one sequence.
        _case("decode_lm_rotary", "module_decode", "bf16", 1, 8, 64, 771, dim=512, tokens=8, prenorm=True, rotary=True),
        # Serving a few long sequences, an odd number of positions.
        _case("decode_b8_8191", "op_decode", "bf16", 8, 16, 128, 8191),
        # The decode benchmark: 64 sequences of 8192 positions, caches of 8.6 GB.
        _case("decode_b64_8192", "op_decode", "bf16", 64, 16, 128, 8192),
        # A short prompt of ragged length through one layer of the language model.
        _case("prefill_lm_197", "module_prefill", "bf16", 1, 8, 64, 197, dim=512, prenorm=True, rotary=True),
        # A long prompt, just short of 64 blocks of 128 positions.
        _case("prefill_8190_d128", "module_prefill", "bf16", 1, 16, 128, 8190, dim=2048),
        # The smallest training step: the reference's own test shape, fp32.
        _case("train_256_fp32", "module_train", "fp32", 2, 2, 64, 256, dim=128),
        # One layer of the byte language model's training step.
        _case("train_lm_layer", "module_train", "bf16", 16, 8, 64, 1024, dim=512, prenorm=True),
        # Ragged, fp16, six tensors instead of the packed projection output.
        _case("train_1333_d128_fp16", "op_train", "fp16", 2, 8, 128, 1333),
        # Scoring without gradients, one position more than 16 blocks.
        _case("forward_b8_2049", "op_forward", "bf16", 8, 16, 64, 2049),
        # The headline benchmark: forward and backward of the core.
        _case("train_b4_4096", "packed_train", "bf16", 4, 16, 64, 4096),
        # The long-context benchmark's share of one GPU.
        _case("train_16384_d128", "packed_train", "bf16", 1, 32, 128, 16384),
    ]


MOST_STEPS = 19 * 32 * 16384 ** 2 * 128        # the largest listed training case
MOST_ELEMENTS = 32 * 16384 * 128               # elements of one of its tensors
MOST_CACHE = 64 * 16 * 8192 * 128 * 2          # bytes of one cache of the largest listed decode case


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["module_decode", "module_prefill", "module_train", "op_decode", "op_forward", "op_train",
                       "packed_train"])
    dtype = rng.choice(["bf16"] * 6 + ["fp16"] * 2 + ["fp32"] * 2)
    dim_head = rng.choice([32, 64, 64, 64, 128, 128])
    heads = _log_uniform(rng, 2, 32)
    module = kind.startswith("module")
    rotary = module and rng.random() < 0.25
    prenorm = module and rng.random() < 0.5
    size = 4 if dtype == "fp32" else 2
    if kind.endswith("decode"):
        batch = _log_uniform(rng, 1, 64)
        n = _log_uniform(rng, 64, 16384)
        while batch * heads * n * dim_head * size > MOST_CACHE:
            batch = (batch + 1) // 2
    else:
        batch = _log_uniform(rng, 1, 16)
        n = _log_uniform(rng, 100, 16384)
        part = 5 if kind.endswith(("forward", "prefill")) else 19
        while (batch * heads * n * max(dim_head, 64) * size > 2 * MOST_ELEMENTS
               or part * batch * heads * n * n * max(dim_head, 64) > MOST_STEPS):
            if batch > 1:
                batch = (batch + 1) // 2
            elif heads > 2:
                heads = (heads + 1) // 2
            else:
                n = n * 3 // 4
    return _case(None, kind, dtype, batch, heads, dim_head, n, dim=heads * dim_head if module else 0,
                 tokens=8 if kind == "module_decode" else 1, prenorm=prenorm, rotary=rotary)


def _randn(shape, dtype, gen, std=1.0):
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=gen)


def _caches(c, dtype, gen, spare):
    """Four (B, H, n + spare, d) buffers with n valid rows.  Rows of qu, kc and vc are projections of unit-variance
    inputs by default-initialised weights (standard deviation 1/sqrt 3); a lookahead key is a sum of about n such
    rows with gates around 1/2, so it grows like sqrt n, and later rows have summed up fewer."""
    B, H, n, d = c["batch"], c["heads"], c["n"], c["dim_head"]
    bufs = [_randn((B, H, n + spare, d), dtype, gen, 3 ** -0.5) for _ in range(4)]
    left = torch.arange(n + spare - 1, -1, -1, device="cuda", dtype=torch.float32)
    bufs[0].mul_((0.25 * left).sqrt().to(dtype)[:, None])
    return bufs


def prepare(case, seed):
    c, dtype = case, DTYPES[case["dtype"]]
    B, H, n, d = c["batch"], c["heads"], c["n"], c["dim_head"]
    gen = torch.Generator("cuda").manual_seed(seed)
    s = {"case": c}
    if c["kind"].startswith("module"):
        torch.manual_seed(seed)
        with torch.device("cuda"):
            s["model"] = Castle(c["dim"], heads=H, dim_head=d, prenorm=c["prenorm"], rotary_emb=c["rotary"])
        s["model"].to(dtype)
    if c["kind"] == "module_decode":
        s["x"] = _randn((B, c["tokens"], c["dim"]), dtype, gen)
        s["bufs"] = _caches(c, dtype, gen, c["tokens"])
    elif c["kind"] == "module_prefill":
        s["x"] = _randn((B, n, c["dim"]), dtype, gen)
    elif c["kind"] == "module_train":
        s["x"] = _randn((B, n, c["dim"]), dtype, gen).requires_grad_()
        s["grad"] = _randn((B, n, c["dim"]), dtype, gen)
    elif c["kind"] == "op_decode":
        s["new"] = [_randn((B, H, 1, d), dtype, gen, 3 ** -0.5) for _ in range(6)]
        s["bufs"] = _caches(c, dtype, gen, 64)
    elif c["kind"] == "packed_train":
        s["packed"] = _randn((B, n, 6, H, d), dtype, gen, 3 ** -0.5).requires_grad_()
        s["grad"] = _randn((B, n, H, d), dtype, gen).permute(0, 2, 1, 3)   # laid out as merging the heads leaves it
    else:
        s["qkv"] = [_randn((B, H, n, d), dtype, gen, 3 ** -0.5) for _ in range(6)]
        if c["kind"] == "op_train":
            for t in s["qkv"]:
                t.requires_grad_()
            s["grad"] = _randn((B, H, n, d), dtype, gen)
    return s


def run(state):
    c = state["case"]
    kind, n, scale = c["kind"], c["n"], c["dim_head"] ** -0.5
    if kind == "module_decode":
        model, x, outs = state["model"], state["x"], []
        with torch.no_grad():
            cache = cache_from_buffers(*state["bufs"], n)
            for i in range(c["tokens"]):
                out, cache = model(x[:, i:i + 1], cache=cache)
                outs.append(out)
        return {"out": outs, "cache": tuple(cache)}
    if kind == "module_prefill":
        with torch.no_grad():
            out, cache = state["model"](state["x"], return_next_cache=True)
        return {"out": out, "cache": tuple(cache)}
    if kind == "module_train":
        model = state["model"]
        out = model(state["x"])
        grads = torch.autograd.grad(out, [state["x"], *model.parameters()], state["grad"])
        return {"out": out.detach(), "grads": grads}
    if kind == "op_decode":
        out = castle_decode_step(*state["new"], *state["bufs"], n, scale)
        return {"out": out, "cache": [b[:, :, :n + 1] for b in state["bufs"]]}
    if kind == "op_forward":
        with torch.no_grad():
            return castle_attention(*state["qkv"], scale)
    if kind == "op_train":
        out = castle_attention(*state["qkv"], scale)
        return {"out": out.detach(), "grads": torch.autograd.grad(out, state["qkv"], state["grad"])}
    out = castle_attention_packed(state["packed"], scale)
    return {"out": out.detach(), "grads": torch.autograd.grad(out, [state["packed"]], state["grad"])}


def work(case):
    """One pass with every input read once and every output written once.  Attention flops in units of one causal
    (n x n) x d product, 2 * n(n+1)/2 * d: forward 5 (gate, state, its use in the scores, scores, P V), backward 10; scores that a backward recomputes count nothing."""
    c = case
    B, H, n, d, dim, tokens = (c[k] for k in ("batch", "heads", "n", "dim_head", "dim", "tokens"))
    size = 4 if c["dtype"] == "fp32" else 2
    inner = H * d
    rows = B * n * inner                       # elements of one (B, H, n, d) tensor
    weights = 7 * dim * inner + (dim if c["prenorm"] else 0)
    if c["kind"].endswith("decode"):
        per_token = 10 * rows + (2 * B * 7 * dim * inner if dim else 0)
        # the four caches in and U out; a row appended to each, the token in and out
        elements = 5 * rows + 4 * tokens * B * inner + weights + tokens * B * (2 * dim if dim else 7 * inner)
        return {"bytes": size * elements, "flops": tokens * per_token}
    unit = B * H * n * (n + 1) * d
    projections = 2 * B * n * 7 * dim * inner
    if c["kind"] == "module_prefill":
        return {"bytes": size * (2 * B * n * dim + weights + 4 * rows), "flops": 5 * unit + projections}
    if c["kind"] == "op_forward":
        return {"bytes": size * 7 * rows, "flops": 5 * unit}
    if c["kind"] == "module_train":
        return {"bytes": size * (4 * B * n * dim + 2 * weights), "flops": 15 * unit + 3 * projections}
    return {"bytes": size * 14 * rows, "flops": 15 * unit}


def tolerance(case):
    """Decode steps compute in fp32 and round what they store.  Parallel passes compute with 16-bit operands whatever
    the caller's type (fp16 for fp32 callers); a gradient goes through several tiles and a long running sum that are
    rounded to 16 bits on the way, and is off by 0.7e-2 (1024 positions) to 1.2e-2 (4096) of its norm in bf16 and by
    1.5e-3 in fp16 (4096) from one computed in fp32: two correct ones differ by up to 1.5 times that."""
    c = case
    if c["kind"].endswith("decode"):
        return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "fp32": 1e-5}[c["dtype"]]}
    if c["kind"].endswith("train"):
        return {"rel": {"bf16": 2e-2, "fp16": 4e-3, "fp32": 4e-3}[c["dtype"]]}
    return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "fp32": 2e-3}[c["dtype"]]}
