"""Timed cases of the operator set: what a user's program has it do, through the modules of
``rgd_triton_b200.ops``, over the range of sizes, types and options it is used with.

``listed()`` are the standing cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare``
makes what a program holds before the call (module with its launch cache, inputs, upstream gradients),
``run`` is one pass, ``work`` the bytes and operations that pass cannot do without, ``tolerance`` how far
another correct implementation of the same precision may be off.

A case with ``train`` true is forward and backward through autograd (the upstream gradient is given, every
input's gradient comes back); with ``train`` false it is the forward alone, as in sampling.
"""
import torch

from rgd_triton_b200 import ops

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
ROW_OPS = ("rms", "rms2", "l2", "l2x2")
TWO_STREAMS = ("rms2", "l2x2")
HEAD_OPS = ("headln", "rope", "lnrope")
MASKED = -1e4       # what a masked position holds in an additive bias
LARGEST_SCORES = 2 * 24 * 4608 * 4608       # B * H * Tq * Tk of the largest attention case


def listed():
    return [
        # Row norms [B, n, c]: the fp32 training step of a small model (latency and launches) ...
        _rows("rms_train_f32", "rms", "f32", True, 4, 256, 1024),
        # ... L2 normalisation of odd-sized embeddings at inference (rows that no vector width divides) ...
        _rows("l2_infer_odd_f16", "l2", "f16", False, 3, 1023, 257),
        # ... and text + image streams of one GPU's share of a joint-attention block, in training.
        _rows("rms2_train_joint_bf16", "rms2", "bf16", True, 2, 512, 3072, n2=4096, c2=3072),
        # Per-head operators on q and k: LayerNorm + partial rotary of a large training batch ...
        _heads("lnrope_train_bf16", "lnrope", "bf16", True, 8, 16, 4096, 4096, 128, False, R=64, cut=4096),
        # ... rotary on the image tokens of a joint sequence while sampling ...
        _heads("rope_infer_joint_bf16", "rope", "bf16", False, 2, 24, 4608, 4608, 128, False, R=64, cut=4096),
        # ... LayerNorm of unequal, ragged query / key lengths in the heads-second layout, in training.
        _heads("headln_train_ragged_f16", "headln", "f16", True, 3, 12, 1000, 203, 64, True),
        # Attention (B, T, h, d): the training step the headline throughput is quoted on ...
        _attn("attn_train_bf16", "bf16", True, 4, 16, 4096, 4096, 128),
        # ... training with a full additive bias, blocks of it masked ...
        _attn("attn_train_bias_f16", "f16", True, 2, 24, 4096, 4096, 64, bias="matrix"),
        # ... training of the joint block: q, k, v as views of one packed projection, padded text keys masked ...
        _attn("attn_train_joint_bf16", "bf16", True, 2, 24, 4608, 4608, 128, bias="padding", packed=True),
        # ... training with a head_dim of its own, ragged length, key padding as a vector ...
        _attn("attn_train_d96_f16", "f16", True, 2, 12, 1100, 1100, 96, bias="vector"),
        # ... causal prefill of a ragged prompt ...
        _attn("attn_prefill_causal_bf16", "bf16", False, 2, 16, 3001, 3001, 128, causal=True),
        # ... and one query per sequence against a long context (decode, pooled cross-attention).
        _attn("attn_decode_bf16", "bf16", False, 4, 16, 1, 4096, 128),
    ]


def _rows(name, op, dtype, train, B, n, c, n2=0, c2=0):
    return {"name": name, "op": op, "dtype": dtype, "train": train, "B": B, "n": n, "c": c, "n2": n2, "c2": c2}


def _heads(name, op, dtype, train, B, H, nq, nk, d, heads_second, R=0, cut=0):
    return {"name": name, "op": op, "dtype": dtype, "train": train, "B": B, "H": H, "nq": nq, "nk": nk, "d": d,
            "heads_second": heads_second, "R": R, "cut": cut}


def _attn(name, dtype, train, B, H, tq, tk, d, bias="none", causal=False, packed=False):
    return {"name": name, "op": "attn", "dtype": dtype, "train": train, "B": B, "H": H, "tq": tq, "tk": tk, "d": d,
            "bias": bias, "causal": causal, "packed": packed}


def _spread(rng, lo, hi):
    """A whole number, uniform over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _channels(rng):
    """Row widths: usually a multiple of 64, sometimes any number."""
    c = _spread(rng, 64, 4096)
    return c if rng.random() < 0.3 else max(64, c // 64 * 64)


def draw(rng):
    kind = rng.choice(("rows", "heads", "attn", "attn"))
    train = rng.random() < 0.5
    if kind == "rows":
        op, dtype = rng.choice(ROW_OPS), rng.choice(("f32", "f16", "bf16"))
        two = op in TWO_STREAMS
        case = _rows("", op, dtype, train, rng.randint(1, 8), _spread(rng, 16, 4608), _channels(rng),
                     _spread(rng, 16, 4608) if two else 0, _channels(rng) if two else 0)
    elif kind == "heads":
        op, dtype = rng.choice(HEAD_OPS), rng.choice(("f32", "f16", "bf16"))
        nq, d = _spread(rng, 16, 4608), rng.choice((32, 64, 64, 96, 128, 128))
        nk = nq if rng.random() < 0.5 else _spread(rng, 16, 4608)
        rotary = op != "headln"
        case = _heads("", op, dtype, train, rng.randint(1, 8), rng.randint(1, 24), nq, nk, d, rng.random() < 0.5,
                      rng.choice((d // 2, d)) if rotary else 0, rng.randint(min(nq, nk) // 2, max(nq, nk)) if rotary else 0)
    else:
        use = rng.choice(("self", "self", "self", "cross", "causal", "few"))
        d, dtype = rng.choice((32, 40, 64, 64, 64, 96, 128, 128, 128)), rng.choice(("f16", "bf16"))
        bias = rng.choice(("none", "none", "vector", "matrix", "padding")) if use in ("self", "cross") else "none"
        largest = LARGEST_SCORES if bias in ("none", "vector") else LARGEST_SCORES // 2
        while True:
            tq, tk = _spread(rng, 64, 4608), _spread(rng, 64, 4608)
            if use in ("self", "causal"):
                tk = tq
            elif use == "few":
                tq, train = _spread(rng, 1, 16), False
            if rng.random() < 0.5:      # half the lengths are round ones
                tq, tk = (tq if use == "few" else (tq + 63) // 64 * 64), (tk + 63) // 64 * 64
            B, H = _spread(rng, 1, 8), rng.randint(1, 24)
            if B * H * tq * tk <= largest:
                break
        case = _attn("", dtype, train, B, H, tq, tk, d, bias, use == "causal",
                     use in ("self", "causal") and rng.random() < 0.5)
    del case["name"]
    return case


def _rotary_table(positions, R, dtype):
    """[2, positions, R]: sin, cos of t * 10000^(-2i/R), each angle repeated for its pair."""
    inv = 1.0 / (10000.0 ** (torch.arange(0, R, 2, dtype=torch.float32, device="cuda") / R))
    ang = (torch.arange(positions, dtype=torch.float32, device="cuda")[:, None] * inv).repeat_interleave(2, dim=-1)
    return torch.stack([ang.sin(), ang.cos()]).to(dtype)


def _bias(case, randn, g, dtype):
    B, H, tq, tk = case["B"], case["H"], case["tq"], case["tk"]
    if case["bias"] == "none":
        return None
    if case["bias"] == "matrix":
        # a learned or positional bias, N(0, 1), with 64 x 64 blocks of it masked; the diagonal stays
        bias = randn(B, H, tq, tk)
        nq, nk = -(-tq // 64), -(-tk // 64)
        blocks = torch.rand(B, H, nq, nk, generator=g, device="cuda") < 0.1
        blocks &= ~torch.eye(nq, nk, dtype=torch.bool, device="cuda")
        blocks[..., 0] = False
        bias.masked_fill_(blocks.repeat_interleave(64, 2)[:, :, :tq].repeat_interleave(64, 3)[..., :tk], MASKED)
        return bias
    # key padding: up to a ninth of the keys, at the end, another number in each sequence
    used = tk - torch.randint(0, tk // 9 + 1, (B,), generator=g, device="cuda")
    masked = torch.arange(tk, device="cuda")[None, :] >= used[:, None]
    bias = torch.zeros(B, 1, 1, tk, device="cuda", dtype=dtype).masked_fill_(masked[:, None, None, :], MASKED)
    return bias if case["bias"] == "vector" else bias.expand(B, H, tq, tk).contiguous()


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype, train, op, B = DTYPES[case["dtype"]], case["train"], case["op"], case["B"]

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)

    state = {"train": train, "op": op, "inputs": [], "grads": [], "rest": ()}
    if op in ROW_OPS:
        shapes = [(B, case["n"], case["c"])] + ([(B, case["n2"], case["c2"])] if op in TWO_STREAMS else [])
        xs = [randn(*s) for s in shapes]
        weights = []
        if op == "rms":
            module = ops.FusedRMSNorm(case["c"], device="cuda", dtype=dtype)
            weights = [module.weight]
        elif op == "rms2":
            module = ops.FusedRMSNorm2((case["c"], case["c2"]), device="cuda", dtype=dtype)
            weights = [module.weight1, module.weight2]
        else:
            module = ops.L2Normalize() if op == "l2" else ops.FusedL2Normalize2()
        with torch.no_grad():
            for w in weights:
                w.copy_(1 + 0.02 * randn(*w.shape))
        state.update(module=module, args=xs, inputs=xs + weights, grads=[randn(*s) for s in shapes])
    elif op in HEAD_OPS:
        H, d = case["H"], case["d"]
        shapes = [(B, H, n, d) if case["heads_second"] else (B, n, H, d) for n in (case["nq"], case["nk"])]
        xs = [randn(*s) for s in shapes]
        if op == "headln":
            module, rest = ops.FusedHeadLayerNorm(), (case["heads_second"], 1e-5)
        else:
            table = _rotary_table(max(case["nq"], case["nk"]) + 1, case["R"], dtype)
            cut = (min(case["cut"], case["nq"]), min(case["cut"], case["nk"]))
            module = ops.RoPE() if op == "rope" else ops.FusedLNRoPE()
            rest = (table, cut, case["heads_second"]) + ((1e-5,) if op == "lnrope" else ())
        state.update(module=module, args=xs, rest=rest, inputs=list(xs), grads=[randn(*s) for s in shapes])
    else:
        H, tq, tk, d = case["H"], case["tq"], case["tk"], case["d"]
        if case["packed"]:
            q, k, v = randn(B, tq, 3, H, d).unbind(2)
        else:
            q, k, v = randn(B, tq, H, d), randn(B, tk, H, d), randn(B, tk, H, d)
        state.update(module=ops.FlashAttention(), args=[q, k, v], rest=(_bias(case, randn, g, dtype), case["causal"]),
                     inputs=[q, k, v], grads=[randn(B, tq, H, d)])
    for t in state["inputs"]:
        t.requires_grad_(train)
    return state


def run(state):
    if not state["train"]:
        with torch.no_grad():
            return state["module"](*state["args"], *state["rest"])
    out = state["module"](*state["args"], *state["rest"])
    outs = list(out) if isinstance(out, (tuple, list)) else [out]
    return outs, list(torch.autograd.grad(outs, state["inputs"], state["grads"]))


def work(case):
    size, train, op, B = DTYPES[case["dtype"]].itemsize, case["train"], case["op"], case["B"]
    if op in ROW_OPS:
        values = B * (case["n"] * case["c"] + case["n2"] * case["c2"])
        weights = case["c"] + case["c2"] if op.startswith("rms") else 0
        # forward x -> y; with the backward also dy -> dx (x is read once for both), w and dw
        return {"bytes": size * (values * (4 if train else 2) + weights * (2 if train else 1)),
                "flops": values * (12 if train else 4)}
    if op in HEAD_OPS:
        values = B * case["H"] * (case["nq"] + case["nk"]) * case["d"]
        table = 2 * (max(case["nq"], case["nk"]) + 1) * case["R"]
        return {"bytes": size * (values * (4 if train else 2) + table), "flops": values * (16 if train else 6)}
    H, tq, tk, d = case["H"], case["tq"], case["tk"], case["d"]
    scores = B * H * tq * tk
    if case["causal"]:      # query i sees keys 0..i
        seen = min(tq, tk)
        scores = B * H * (seen * (seen + 1) // 2 + (tq - seen) * tk)
    bias = {"none": 0, "vector": B * tk, "matrix": B * H * tq * tk, "padding": B * H * tq * tk}[case["bias"]]
    rows = B * H * d * (2 * tq + 2 * tk)                            # q, k, v -> o
    if train:
        rows += B * H * d * (2 * tq + 2 * tk)                       # dO -> dq, dk, dv
    # 2 products of 2 * scores * d operations forward, 5 in the backward
    return {"bytes": size * (rows + bias), "flops": 4 * scores * d * (3.5 if train else 1)}


def tolerance(case):
    # one rounding of the outputs; attention also rounds the probabilities that it multiplies by
    return {"rel": {"f32": 1e-5, "f16": 2e-3, "bf16": 1e-2}[case["dtype"]]}
