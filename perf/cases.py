"""What users of this framework have it do, as cases that can be timed.

A case names a use of the operator (``use``), the geometry and the data type; ``prepare`` makes what the
caller holds before the call, ``run`` makes one pass through the public entry points, ``work`` counts what
the pass cannot do without.  ``listed`` holds the reference points, ``draw`` gives more of the same ranges.

Uses:
  call     ``oal_attention`` on tensors without gradients: the one-call form, groups validated every time
  infer    ``run_prepared_grouped_hd_block_gemm`` without gradients: prompt processing with a kept plan
  train    the prepared call with gradients, forward + backward, every launch queued from Python
  replay   forward + backward of a prepared call as a recorded step, on new values in every pass
  layer    a decoder layer's attention block (projections with low-rank updates, rotary embedding,
           operator, output projection), forward + backward
"""

from __future__ import annotations

import math

import torch

from oal_b200 import oal_attention, prepare_grouped_hd_block_gemm, run_prepared_grouped_hd_block_gemm
from oal_b200.attention_shell import ModelGeometry, OalAttentionLayer, PreparedCallCache, rope_tables
from oal_b200.captured_step import CapturedStep
from oal_b200.synthetic import QWEN_GROUP_SIZES

# group sizes of the configured partitions; other counts are cut evenly
_SIZES = dict(QWEN_GROUP_SIZES)


def _case(name, use, b, n, *, hq=14, hkv=2, d=64, g=8, dtype="bfloat16", per_head=False, aux=False):
    c = dict(use=use, b=b, n=n, hq=hq, hkv=hkv, d=d, g=g, dtype=dtype, per_head=per_head, aux=aux)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one short prompt scored with the one-call API: latency of validation, launches and the status read
        _case("call_n200", "call", 1, 200),
        # a short training sequence, launch-bound from Python
        _case("train_n256", "train", 1, 256),
        # the sweep's shortest sequence: eager, and recorded as a graph (the documented way to run it)
        _case("train_n1024", "train", 1, 1024),
        _case("replay_n1024", "replay", 1, 1024),
        # prompt processing of a batch at the model's context length
        _case("infer_b4_n4096", "infer", 4, 4096),
        # the benchmark's workload: forward + backward of a batch of four at 4096 tokens
        _case("train_b4_n4096", "train", 4, 4096),
        # the sweep's longest sequence
        _case("train_n65536", "train", 1, 65536),
        # the finest partition of the sweep (sixteen groups of four dimensions)
        _case("train_g16_n4096", "train", 1, 4096, g=16),
        # odd length and batch, heads narrower than 64, a partition per head, gradients of all three outputs
        _case("train_ragged_b3_n1999", "train", 3, 1999, hq=8, hkv=4, d=48, g=4, per_head=True, aux=True),
        # an attention block inside the model-level training step: batch 8 at 4096 tokens per GPU
        _case("layer_b8_n4096", "layer", 8, 4096, per_head=True),
        # exact fp32 mode: the configured small check case, and a full-width layer for parity runs
        _case("exact_n256", "train", 1, 256, hq=2, hkv=2, g=4, dtype="float32"),
        _case("exact_n2048", "train", 1, 2048, dtype="float32"),
    ]


def draw(rng):
    def length(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return n if rng.random() < 0.5 else max(lo, min(hi, (n + 63) // 64 * 64))

    r = rng.random()
    g = rng.choice((1, 2, 4, 6, 8, 8, 8, 12, 16))
    heads = rng.choice(((14, 2), (14, 2), (14, 2), (8, 4), (16, 2), (4, 4), (7, 1), (2, 2)))
    hq, hkv = heads
    d = rng.choice((64, 64, 64, 64, 48, 32))
    per_head = rng.random() < 0.5
    if r < 0.15:
        return _case(None, "call", rng.choice((1, 1, 2)), length(16, 2048), hq=hq, hkv=hkv, d=d, g=g, per_head=per_head)
    if r < 0.32:
        n = length(128, 16384)
        return _case(None, "infer", max(1, min(rng.randint(1, 8), 16384 // n)), n, hq=hq, hkv=hkv, d=d, g=g,
                     per_head=per_head)
    if r < 0.62:
        n = length(64, 32768 if g <= 8 else 8192)
        return _case(None, "train", max(1, min(rng.randint(1, 8), 16384 // n)), n, hq=hq, hkv=hkv, d=d, g=g,
                     per_head=per_head, aux=rng.random() < 0.25)
    if r < 0.76:
        return _case(None, "replay", rng.randint(1, 2), length(64, 2048), hq=hq, hkv=hkv, d=d, g=g, per_head=per_head)
    if r < 0.86:
        n = length(256, 8192)
        return _case(None, "layer", max(1, min(rng.randint(1, 8), 16384 // n)), n, g=rng.choice((4, 8, 8)), per_head=True)
    dtype = rng.choice(("float32", "float32", "float16"))
    return _case(None, rng.choice(("train", "train", "infer")), rng.choice((1, 1, 2)), length(32, 1448), hq=hq, hkv=hkv,
                 d=d, g=g, dtype=dtype, per_head=per_head)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _groups(case, gen):
    """Seeded partitions of the head dimension: int32 [d], or [hq, d] with one partition per query head."""
    d, g = case["d"], case["g"]
    sizes = _SIZES.get(g) if d == 64 else None
    if sizes is None:
        sizes = [d // g + (i < d % g) for i in range(g)]
    ids = torch.repeat_interleave(torch.arange(g), torch.tensor(sizes)).to(torch.int32)
    rows = [ids[torch.randperm(d, generator=gen)] for _ in range(case["hq"] if case["per_head"] else 1)]
    return torch.stack(rows) if case["per_head"] else rows[0]


def _tensors(case, seed):
    """q, k with a few outlier channels, v and the upstream gradients ~ N(0, 1); packed factors ~ U(0.1, 1)."""
    dev, dtype = torch.device("cuda"), getattr(torch, case["dtype"])
    cpu = torch.Generator().manual_seed(seed)
    gen = torch.Generator(device=dev).manual_seed(seed)
    b, n, hq, hkv, d, g = (case[x] for x in ("b", "n", "hq", "hkv", "d", "g"))
    gain = torch.ones(d)
    gain[torch.randperm(d, generator=cpu)[:4]] = OUTLIER_GAIN if g >= 4 else OUTLIER_GAIN_COARSE
    gain = gain.to(dev)

    def normal(h, scale=None):
        t = torch.randn(b, h, n, d, generator=gen, device=dev)
        return (t if scale is None else t * scale).to(dtype)

    p = (g + 1) * (g + 2) // 2
    return dict(q=normal(hq, gain), k=normal(hkv, gain), v=normal(hkv), dout=normal(hq),
                groups=_groups(case, cpu).to(dev), factor=(torch.rand(hq, p, generator=cpu) * 0.9 + 0.1).to(dev), gen=gen)


# the outlier channels of attention queries and keys: four of them, this many times the others' deviation.
# A partition exists to keep them apart: with one or two groups they share a group, where gains this large leave
# the coefficient gradient a difference of terms a thousand times its size, which bf16 inputs do not determine.
OUTLIER_GAIN = 20.0
OUTLIER_GAIN_COARSE = 4.0


def prepare(case, seed):
    use = case["use"]
    if use == "layer":
        return _prepare_layer(case, seed)
    t = _tensors(case, seed)
    q, k, v, groups, factor, dout = t["q"], t["k"], t["v"], t["groups"], t["factor"], t["dout"]
    precision = "bf16_tensorcore" if case["dtype"] == "bfloat16" else "fp32_ieee"
    if use == "call":
        return dict(use=use, q=q, k=k, v=v, groups=groups, factor=factor)
    if use == "infer":
        prepared = prepare_grouped_hd_block_gemm(q, k, v, groups, factor, precision=precision)
        return dict(use=use, q=q, k=k, v=v, factor=factor, prepared=prepared)
    leaves = [x.requires_grad_() for x in (q, k, v, factor)]
    prepared = prepare_grouped_hd_block_gemm(q, k, v, groups, factor, precision=precision)
    if use == "replay":
        values = [x.detach() for x in leaves] + [dout]
        return dict(use=use, values=values, step=CapturedStep(prepared, q, k, v, factor, dout))
    grads = [dout]
    if case["aux"]:        # the numerator and the denominator are outputs of the operator too
        grads.append(0.1 * torch.randn(dout.shape, generator=t["gen"], device=dout.device))
        grads.append(0.1 * torch.randn(dout.shape[:3] + (1,), generator=t["gen"], device=dout.device))
    return dict(use=use, leaves=leaves, prepared=prepared, grads=grads)


def _prepare_layer(case, seed):
    dev, dtype = torch.device("cuda"), getattr(torch, case["dtype"])
    cpu = torch.Generator().manual_seed(seed)
    gen = torch.Generator(device=dev).manual_seed(seed)
    b, n, hq, g = case["b"], case["n"], case["hq"], case["g"]
    geometry = ModelGeometry(num_query_heads=hq, num_kv_heads=case["hkv"], hidden_size=hq * case["d"], head_dim=case["d"])
    factor = torch.rand(hq, (g + 1) * (g + 2) // 2, generator=cpu) * 0.9 + 0.1
    layer = OalAttentionLayer(0, _groups(case, cpu), factor, cache=PreparedCallCache(output_layout="tokens_first"),
                              geometry=geometry, dtype=dtype).to(dev)
    with torch.no_grad():
        for name, p in layer.named_parameters():
            if name != "factor":      # projections, biases and low-rank matrices of a trained scale
                p.copy_(torch.randn(p.shape, generator=gen, device=dev) * 0.04)
    shape = (b, n, geometry.hidden_size)
    x = torch.randn(shape, generator=gen, device=dev).to(dtype).requires_grad_()
    dout = torch.randn(shape, generator=gen, device=dev).to(dtype)
    return dict(use="layer", layer=layer, x=x, dout=dout, rope=rope_tables(n, case["d"], device=dev),
                leaves=[x] + [p for p in layer.parameters() if p.requires_grad])


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    use = state["use"]
    if use == "call":
        return oal_attention(state["q"], state["k"], state["v"], state["groups"], state["factor"])
    if use == "infer":
        return run_prepared_grouped_hd_block_gemm(state["prepared"], state["q"], state["k"], state["v"], state["factor"])
    if use == "replay":
        return state["step"].replay(*state["values"])
    for leaf in state["leaves"]:
        leaf.grad = None
    if use == "layer":
        out = state["layer"](state["x"], state["rope"])
        out.backward(state["dout"])
        return [out.detach()] + [leaf.grad for leaf in state["leaves"]]
    outs = run_prepared_grouped_hd_block_gemm(state["prepared"], *state["leaves"])
    grads = state["grads"]
    torch.autograd.backward(outs[:len(grads)], grads)
    return [o.detach() for o in outs] + [leaf.grad for leaf in state["leaves"]]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    b, n, hq, hkv, d, g = (case[x] for x in ("b", "n", "hq", "hkv", "d", "g"))
    size = torch.empty((), dtype=getattr(torch, case["dtype"])).element_size()
    backward = case["use"] in ("train", "replay", "layer")
    # forward contractions by the cheaper of the two exact statements: token pairs (scores, weight x values), or
    # the running state over 1 + d + d (d + 1) / 2 features (update per KV head, read per query head); every
    # contraction has two transposes in the backward
    features, e = 1 + d + d * (d + 1) // 2, d + 1
    pairs = hq * (n * (n + 1) // 2) * 2 * (d + e)
    scan = n * (hq + hkv) * 2 * features * e
    flops = b * min(pairs, scan) * (3 if backward else 1)
    tokens = b * n
    qkv, outs = tokens * (hq + 2 * hkv) * d * size, tokens * hq * d * size
    moved = qkv + outs + (0 if case["use"] == "call" else 4 * tokens * hq * e)     # out; numerator and denominator in fp32
    if backward:
        moved += outs + qkv                                                        # upstream gradient; dq, dk, dv
        if case["aux"]:
            moved += 4 * tokens * hq * e
    if case["use"] == "replay":
        moved = 2 * (qkv + outs)
    if case["use"] == "layer":
        hidden = hq * d
        # four projections with rank-16 updates; frozen weights: one product forward, one backward each
        flops += 2 * tokens * 2 * (2 * hidden * hidden + 2 * hidden * hkv * d)
        flops += 3 * tokens * 2 * 16 * (2 * (hidden + hidden) + 2 * (hidden + hkv * d))
        moved = 4 * tokens * hidden * size + 2 * 2 * (2 * hidden * hidden + 2 * hidden * hkv * d)
    return {"bytes": int(moved), "flops": int(flops)}


def tolerance(case):
    if case["dtype"] == "bfloat16":
        # gradients chain twice as many bf16-rounded operands, and the coefficient gradient cancels
        return {"rel": 1e-2 if case["use"] in ("call", "infer") else 2e-2}
    if case["dtype"] == "float16":
        return {"rel": 1e-3}
    return {"rel": 1e-5}
