"""Performance cases of the attention kernels: what a user of this package runs, through its public
entry points, over the range of sizes, masks and data types that the path is used with.

Passes:
  forward   `flash_attention_v7` without gradients (evaluation, prefill)
  train     forward and first backward (ordinary training)
  second    forward, backward with `create_graph`, double backward: one use of attention in a
            test-time-training step, whose outer loss is differentiated through an inner gradient
  hvp       `attention_cuda.v7_double_backward` alone, with O and L from an earlier forward: the
            Hessian-vector product that bench.py times
  prep      `qk_norm_rope` without gradients: RMS norm + rotary embedding + layout change of a
            Q or K projection, in front of attention
  prep_train   the same with its backward (gradients of x and of the norm's weight)

A case of the attention passes is [B, H, N_q, D] queries against [B, H, N_kv, D] keys with the
chunked causal sliding-window mask (`window`, `chunk`), or no mask (`mask_mode` 1); `amp` is the
standard deviation of Q and K (2 gives peaked softmax rows).
"""
import importlib
import math

import torch

attention = importlib.import_module("610sample_b200.attention")
attention_cuda = importlib.import_module("610sample_b200.attention_cuda")
qk_prep = importlib.import_module("610sample_b200.qk_prep")

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _attn(name, do, B, H, N_q, N_kv, D, window, chunk, dtype="bf16", mask_mode=0, amp=1.0):
    c = dict(do=do, B=B, H=H, N_q=N_q, N_kv=N_kv, D=D, window=window, chunk=chunk, dtype=dtype,
             mask_mode=mask_mode, amp=amp)
    return dict(name=name, **c) if name else c


def _prep(name, do, n_tok, H, D, dtype="bf16"):
    c = dict(do=do, n_tok=n_tok, H=H, D=D, dtype=dtype)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # the small shape of bench_attn_meta.py: a second-order step on short chunks, where launches
        # and host work are most of the time
        _attn("second_small_64x256", "second", 1, 4, 64, 256, 64, 192, 2),
        # the fp32 reference configuration (B2 H4 N256 D64, causal): gradient checks and debugging
        _attn("second_fp32_256", "second", 2, 4, 256, 256, 64, 256, 0, "fp32"),
        # odd sizes, fp16: sequences that are no multiple of any tile, keys with a history, as in
        # training on packed documents
        _attn("train_fp16_ragged", "train", 2, 12, 777, 1301, 80, 1000, 1, "fp16"),
        # evaluation of the 760M shape: one chunk of 1024 queries against a full window of keys
        _attn("forward_chunk_760M", "forward", 1, 16, 1024, 9216, 96, 8192, 8),
        # one chunk of the 125M shape early in the sequence, half of the window still empty
        _attn("second_chunk_125M", "second", 1, 12, 1024, 9216, 64, 8192, 3),
        # a late chunk of the 3B shape, the largest of the sliding-window models
        _attn("second_chunk_3B", "second", 1, 32, 1024, 9216, 80, 8192, 7),
        # one layer of the end-to-end step of bench_ttt.py (batch 8, 12 heads, sequence 2048)
        _attn("second_ttt_2048", "second", 8, 12, 2048, 2048, 64, 2048, 0),
        # no mask: encoder-style attention, first order
        _attn("train_nomask_2048", "train", 4, 16, 2048, 2048, 64, 2048, 0, "bf16", 1, 0.5),
        # the headline workload of bench.py
        _attn("hvp_4096", "hvp", 4, 16, 4096, 4096, 128, 4096, 0),
        # long context, peaked rows: the largest case
        _attn("second_long_16384", "second", 1, 32, 16384, 16384, 128, 16384, 0, "bf16", 0, 2.0),
        # norm + rotary embedding of the key stream of the 125M shape
        _prep("prep_9216x12x64", "prep", 9216, 12, 64),
        # the same step in training, at the token count of the end-to-end step
        _prep("prep_train_2048x12x64", "prep_train", 2048, 12, 64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


_LARGEST = 2.2e13      # operations of the largest listed case, rounded up


def draw(rng):
    kind = rng.choice(["small", "causal", "causal", "chunk", "chunk", "nomask", "fp32", "prep"])
    half = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "small":
        N_q = _log_int(rng, 32, 256)
        N_kv = int(N_q * rng.uniform(1.0, 4.0))
        return _attn(None, rng.choice(["forward", "train", "second"]), rng.randint(1, 2), rng.randint(1, 8), N_q, N_kv,
                     rng.choice([64, 80, 96, 128]), _log_int(rng, 32, N_kv), rng.randint(0, 4), half)
    if kind == "fp32":
        N = _log_int(rng, 128, 1024)
        return _attn(None, rng.choice(["train", "second"]), rng.randint(1, 2), rng.randint(2, 8), N, N,
                     rng.choice([64, 80, 128]), N, 0, "fp32")
    if kind == "prep":
        return _prep(None, rng.choice(["prep", "prep_train"]), _log_int(rng, 256, 16384), rng.choice([8, 12, 16, 32]),
                     rng.choice([64, 80, 96, 128]), half)
    while True:
        do = rng.choice(["forward", "train", "second", "second", "hvp"])
        if kind == "chunk":       # chunks of a sliding-window model: N_q new tokens, window + N_q keys
            N_q = _log_int(rng, 256, 2048)
            window = _log_int(rng, 1024, 8192)
            c = _attn(None, do, rng.randint(1, 4), rng.choice([8, 12, 16, 32]), N_q, N_q + window,
                      rng.choice([64, 80, 96, 128]), window, rng.randint(0, 8), half)
        elif kind == "causal":    # plain causal attention over N tokens
            N = _log_int(rng, 512, 16384)
            c = _attn(None, do, rng.randint(1, 8), rng.choice([8, 12, 16, 32]), N, N, rng.choice([64, 64, 96, 128, 128]),
                      N, 0, half, 0, rng.choice([1.0, 1.0, 2.0]))
        else:                     # no mask: encoders and cross attention
            N = _log_int(rng, 256, 4096)
            N_kv = rng.choice([N, N, _log_int(rng, 256, 4096)])
            c = _attn(None, do, rng.randint(1, 4), rng.choice([8, 16]), N, N_kv, rng.choice([64, 128]), N_kv, 0, half, 1, 0.5)
        if work(c)["flops"] <= _LARGEST and work(c)["bytes"] <= 4e9:
            return c


def _visible_pairs(c):
    """(query, key) pairs of one head that the mask lets through."""
    N_q, N_kv = c["N_q"], c["N_kv"]
    if c["mask_mode"]:
        return N_q * N_kv
    q0, k0 = c["chunk"] * N_q, c["chunk"] * N_q + N_q - N_kv
    n = 0
    for i in range(N_q):
        lo = max(0, k0, q0 + i - c["window"] + 1)
        hi = min(q0 + i, k0 + N_kv - 1)
        n += max(0, hi - lo + 1)
    return n


def work(case):
    c = case
    size = 4 if c["dtype"] == "fp32" else 2
    if c["do"].startswith("prep"):
        n = c["n_tok"] * c["H"] * c["D"]
        table = c["n_tok"] * c["D"] * 4
        # forward: x in, y out.  Backward: x and the gradient of y in, the gradient of x out.
        return {"bytes": (2 if c["do"] == "prep" else 5) * n * size + table, "flops": (8 if c["do"] == "prep" else 24) * n}
    BH = c["B"] * c["H"]
    q, kv, rows = BH * c["N_q"] * c["D"] * size, BH * c["N_kv"] * c["D"] * size, BH * c["N_q"] * 4
    fwd = 2 * q + 2 * kv + rows                  # Q, K, V -> O, L
    bwd = 4 * q + 4 * kv + rows                  # Q, dO, O, K, V, L -> dQ, dK, dV
    hvp = 6 * q + 6 * kv + rows                  # Q, dO, O, g_dQ, K, V, g_dK, g_dV, L -> g_dO, g_Q, g_K, g_V
    products = {"forward": 2, "train": 7, "second": 19, "hvp": 12}[c["do"]]
    moved = {"forward": fwd, "train": fwd + bwd, "second": fwd + bwd + hvp, "hvp": hvp}[c["do"]]
    return {"bytes": moved, "flops": 2 * products * c["D"] * _visible_pairs(c) * BH}


def tolerance(case):
    # half-precision operands and outputs: the rounding of P and dS (2^-9 or 2^-12) and of the results
    return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "fp32": 1e-5}[case["dtype"]]}


def prepare(case, seed):
    c = case
    dt = _DTYPES[c["dtype"]]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def randn(*shape, amp=1.0):
        return (torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32) * amp).to(dt)

    if c["do"].startswith("prep"):
        s = dict(do=c["do"], x=randn(c["n_tok"], c["H"], c["D"]), w=(1.0 + randn(c["D"], amp=0.1)).to(dt),
                 freqs=qk_prep.rope_table(c["D"], c["n_tok"], device="cuda"))
        if c["do"] == "prep_train":
            s["g"] = randn(1, c["H"], c["n_tok"], c["D"])
            s["x"].requires_grad_(True)
            s["w"].requires_grad_(True)
        return s
    qs, ks = (c["B"], c["H"], c["N_q"], c["D"]), (c["B"], c["H"], c["N_kv"], c["D"])
    s = dict(do=c["do"], args=(c["window"], c["chunk"], c["mask_mode"]))
    s["Q"], s["K"], s["V"] = randn(*qs, amp=c["amp"]), randn(*ks, amp=c["amp"]), randn(*ks)
    if c["do"] != "forward":
        s["dO"] = randn(*qs)
    if c["do"] in ("second", "hvp"):
        s["tangents"] = (randn(*qs), randn(*ks), randn(*ks))
    if c["do"] == "hvp":
        s["O"], s["L"] = attention_cuda.v7_forward(s["Q"], s["K"], s["V"], *s["args"])
    elif c["do"] != "forward":
        for n in ("Q", "K", "V"):
            s[n].requires_grad_(True)
        if c["do"] == "second":
            s["dO"].requires_grad_(True)
    return s


def run(state):
    s = state
    do = s["do"]
    if do == "prep":
        return qk_prep.qk_norm_rope(s["x"], s["w"], s["freqs"])
    if do == "prep_train":
        y = qk_prep.qk_norm_rope(s["x"], s["w"], s["freqs"])
        gx, gw = torch.autograd.grad(y, [s["x"], s["w"]], s["g"])
        return y, gx, gw
    if do == "hvp":
        g_dO, g_Q, g_K, g_V = attention_cuda.v7_double_backward(*s["tangents"], s["dO"], s["Q"], s["K"], s["V"],
                                                                s["O"], s["L"], *s["args"])
        return g_dO, g_Q, g_K, g_V
    O = attention.flash_attention_v7(s["Q"], s["K"], s["V"], *s["args"])
    if do == "forward":
        return O
    dQ, dK, dV = torch.autograd.grad(O, [s["Q"], s["K"], s["V"]], s["dO"], create_graph=do == "second")
    if do == "train":
        return O, dQ, dK, dV
    second = torch.autograd.grad([dQ, dK, dV], [s["dO"], s["Q"], s["K"], s["V"]], s["tangents"])
    return (O, dQ, dK, dV) + tuple(second)
