"""The calls whose speed matters to a user of this package, as one list of cases with seeded inputs.

Every case is one call (or one replay of a recorded call) of a public operator, with what a serving program has in hand
before it: queries, paged caches, block table, weights and output buffers on the GPU. Three families:

  decode / prefill  the fused chain indexer -> top-2048 -> sparse attention, one to four query tokens per sequence or a
                    chunk of one prompt
  indexer, attention, prolog  the operators of that chain on their own, as the example drivers call them
  layer             the non-quantised chain with both of its prologs

`graph` cases replay a recorded call (`CapturedCall`), as a decode loop of fixed batch does; the others call the operator
from Python. Sizes are the five benchmark configurations, the batches of the tests, and odd ones between them.
"""
import math
import random

import torch

import pypto_b200 as pto
from pypto_b200 import inputs as gen

TOPK = gen.TOPK
SCALE = 576 ** -0.5
BF16 = torch.bfloat16
DTYPES = {"f16": torch.float16, "f32": torch.float32}


def listed():
    return [
        # one user, short context, called from Python: launches and host work are what counts. fp16 scales are what the
        # quantised prolog produces
        dict(name="decode_1x4k", op="decode", b=1, s1=1, lo=4001, hi=4001, scales="f16", graph=False),
        # the headline configuration: 64 sequences of 4096 to 65536 keys, step recorded once and replayed
        dict(name="decode_64x64k", op="decode", b=64, s1=1, lo=4096, hi=65536, scales="f32", graph=True),
        # speculative decoding at the longest context, two query tokens per sequence
        dict(name="decode_mtp_128x128k", op="decode", b=128, s1=2, lo=131072, hi=131072, scales="f32", graph=False),
        # one chunk of a long prompt: 4096 query tokens at the end of 131072 keys, all heads on this GPU
        dict(name="prefill_4096x128k", op="decode", b=1, s1=4096, lo=131072, hi=131072, scales="f32", graph=False),
        # the indexer alone, indices in order of score
        dict(name="indexer_8x32k", op="indexer", b=8, s1=1, lo=32768, hi=32768, scales="f32", graph=False),
        # the attention alone, smallest published configuration
        dict(name="attention_2x8k", op="attention", layout="split", heads=128, b=2, s1=1, lo=8192, hi=8192, graph=False),
        # the attention over packed 656-byte rows, an odd batch of ragged sequences, some shorter than the selection
        dict(name="attention_packed_33x20k", op="attention", layout="packed", heads=128, b=33, s1=1, lo=1000, hi=20001,
             graph=False),
        # a GPU's share of that prompt chunk when eight GPUs divide the heads: 16 heads for every token
        dict(name="attention_heads16_4096", op="attention", layout="split", heads=16, b=1, s1=4096, lo=131072, hi=131072,
             graph=False),
        # the prolog of a few decoding users, called from Python
        dict(name="prolog_3", op="prolog", b=3, s1=1, graph=False),
        # the prolog of the headline batch, recorded and replayed
        dict(name="prolog_64", op="prolog", b=64, s1=1, graph=True),
        # the prolog of a prompt chunk
        dict(name="prolog_1000", op="prolog", b=1, s1=1000, graph=False),
        # a whole non-quantised layer: both prologs, bf16 indexer, top-k, attention over the bf16 cache
        dict(name="layer_bf16_16x8k", op="layer", b=16, s1=1, lo=4096, hi=8200, graph=False),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["decode", "decode", "prefill", "indexer", "attention", "prolog", "layer"])
    graph = rng.random() < 0.5
    if op == "prefill":
        s1 = _log_int(rng, 64, 4096)
        ctx = _log_int(rng, s1, 131072)
        return dict(op="decode", b=1, s1=s1, lo=ctx, hi=ctx, scales=rng.choice(["f16", "f32"]), graph=False)
    if op == "prolog":
        if rng.random() < 0.7:
            return dict(op="prolog", b=_log_int(rng, 1, 128), s1=rng.choice([1, 1, 2]), graph=graph)
        return dict(op="prolog", b=1, s1=_log_int(rng, 100, 1500), graph=False)
    hi = _log_int(rng, 200, 8192 if op == "layer" else 131072)
    lo = rng.randint(max(1, hi // 16), hi)
    s1 = rng.choice([1, 1, 1, 2, 3, 4])
    # the largest product is that of 128 sequences of 131072 keys with two query tokens
    b = min(_log_int(rng, 1, 32 if op == "layer" else 128), (1 << 25) // (hi * s1))
    case = dict(op=op, b=b, s1=s1, lo=lo, hi=hi, graph=graph)
    if op in ("decode", "indexer"):
        case["scales"] = rng.choice(["f16", "f32"])
    if op == "attention":
        case["layout"] = rng.choice(["split", "packed", "bf16"])
        case["heads"] = rng.choice([128, 128, 16, 32, 64]) if case["layout"] == "split" else 128
    return case


def _lengths(case):
    """Sequence lengths, uniform in [lo, hi] and the same for every seed: they are part of the case's size."""
    r = random.Random("%d %d %d" % (case["b"], case["lo"], case["hi"]))
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["b"])]


# --- inputs -----------------------------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 11)
    return g


def _uni(g, shape, lo, hi, dtype=BF16):
    return torch.empty(shape, dtype=torch.float32, device="cuda").uniform_(lo, hi, generator=g).to(dtype)


def _int8(g, shape, lo=-127):
    return torch.randint(lo, 128, shape, dtype=torch.int8, device="cuda", generator=g)


def _selection(lens, s1, g):
    """Selected positions as an indexer leaves them: per token 2048 distinct positions of its causal range, spread over
    it and in no order; shorter ranges whole, then -1."""
    eff = torch.tensor([max(s - (s1 - 1 - i), 0) for s in lens for i in range(s1)], dtype=torch.int64, device="cuda")[:, None]
    n = eff.clamp(max=TOPK)
    i = torch.arange(TOPK, dtype=torch.int64, device="cuda")[None, :]
    lo = i * eff // n.clamp(min=1)
    hi = (i + 1) * eff // n.clamp(min=1)
    u = torch.rand((eff.shape[0], TOPK), generator=g, device="cuda")
    pos = lo + torch.minimum((u * (hi - lo)).to(torch.int64), hi - lo - 1)
    pos = torch.where(i < n, pos, -1)
    order = (torch.rand(pos.shape, generator=g, device="cuda") + 2 * (i >= n)).argsort(dim=1)
    return pos.gather(1, order).to(torch.int32).contiguous()


def _call(case, op, *args, **kwargs):
    """The state's call: a recorded step to replay, or the operator with its arguments."""
    if case["graph"]:
        return pto.CapturedCall(op, *args, **kwargs).replay
    return lambda: op(*args, **kwargs)


def _prepare_decode(case, seed):
    d = gen.make_inputs(_lengths(case), s1=case["s1"], seed=seed, device="cuda", scale_dtype=DTYPES[case["scales"]])
    idx = torch.zeros((d.t, 1, TOPK), dtype=torch.int32, device="cuda")
    out = torch.zeros((d.b, d.s1, 128, 512), dtype=BF16, device="cuda")
    call = _call(case, pto.decode_indexer_attention_quant, d.idx_query, d.idx_query_scale, d.idx_key_cache,
                 d.idx_key_scale, d.idx_weight, d.query_nope, d.query_rope, d.key_nope_2d, d.key_rope_2d,
                 d.k_nope_scales, d.act_seq_key, d.block_table, idx, out)
    # the selection that the chain leaves in `idx` is a set: its order means nothing and is not the same twice
    return dict(call=call, out=out, keep=(d, idx))


def _prepare_indexer(case, seed):
    d = gen.make_inputs(_lengths(case), s1=case["s1"], seed=seed, device="cuda", scale_dtype=DTYPES[case["scales"]],
                        with_attention=False)
    idx = torch.zeros((d.t, 1, TOPK), dtype=torch.int32, device="cuda")
    call = _call(case, pto.lightning_indexer_decode, d.idx_query, d.idx_query_scale, d.idx_key_cache, d.idx_key_scale,
                 d.idx_weight, d.act_seq_key, d.block_table, idx)
    return dict(call=call, out=idx, keep=d)


def _prepare_attention(case, seed):
    g = _gen(seed)
    lens = _lengths(case)
    heads = case["heads"]
    if case["layout"] == "bf16":
        d = gen.make_nonquant_inputs(lens, s1=case["s1"], seed=seed, device="cuda")
    else:
        d = gen.make_inputs(lens, s1=case["s1"], seed=seed, device="cuda", with_indexer=False, attn_heads=heads)
    sel = _selection(lens, case["s1"], g)
    out = torch.zeros((d.b, d.s1, heads, 512), dtype=BF16, device="cuda")
    tail = (sel, d.block_table, d.act_seq_key, out, heads, 1, SCALE, TOPK, 128, d.max_blocks)
    if case["layout"] == "packed":
        rows = torch.empty((d.block_num * 128, gen.PACKED_ROW_BYTES), dtype=torch.int8, device="cuda")
        pto.pack_kv_cache(d.key_nope_2d, d.key_rope_2d, d.k_nope_scales, rows)
        call = _call(case, pto.sparse_attention_antiquant_d, d.query_nope, d.query_rope, rows, *tail)
    else:
        op = pto.sparse_flash_attention_quant_d if case["s1"] <= 4 else pto.sparse_flash_attention_quant_p
        call = _call(case, op, d.query_nope, d.query_rope, d.key_nope_2d, d.key_rope_2d, d.k_nope_scales, *tail)
    return dict(call=call, out=out, keep=d)


def _new_rows(b, s1, lens, table):
    """Paged row of each new token: the last s1 positions of its sequence."""
    pos = (torch.tensor(lens, dtype=torch.int64, device="cuda")[:, None] - s1
           + torch.arange(s1, dtype=torch.int64, device="cuda")[None, :])
    page = table.to(torch.int64).gather(1, pos // 128)
    return (page * 128 + pos % 128).reshape(b * s1).contiguous()


def _prolog_weights(g, quant):
    """One layer's weights, from the distributions of the example drivers."""
    w = dict(
        w_dq=_uni(g, (gen.HIDDEN, gen.Q_LORA), -0.1, 0.1),
        w_uk=_uni(g, (gen.ATT_HEADS, gen.NOPE_DIM, gen.KV_LORA), -0.1, 0.1),
        w_dkvkr=_uni(g, (gen.HIDDEN, gen.KV_LORA + gen.ROPE_DIM), -0.1, 0.1),
        gamma_cq=_uni(g, (gen.Q_LORA,), -1, 1),
        gamma_ckv=_uni(g, (gen.KV_LORA,), -1, 1),
        ln_gamma=_uni(g, (gen.IDX_DIM,), 0.5, 1.5),
        ln_beta=_uni(g, (gen.IDX_DIM,), -0.5, 0.5),
    )
    up = gen.ATT_HEADS * (gen.NOPE_DIM + gen.ROPE_DIM)
    idx = gen.IDX_HEADS * gen.IDX_DIM
    if quant:
        f = _uni(g, (gen.Q_LORA, up), -0.1, 0.1, torch.float32)
        peak = f.abs().amax(dim=0, keepdim=True)
        w.update(w_uqqr=torch.round(f * (127.0 / peak)).to(torch.int8), w_qb_scale=(peak / 127.0).reshape(-1, 1).contiguous(),
                 w_idx_qb=_int8(g, (gen.Q_LORA, idx), -128), w_idx_qb_scale=_uni(g, (idx, 1), -1, 1, torch.float32),
                 w_idx_k=_uni(g, (gen.HIDDEN, gen.IDX_DIM), -1, 1), w_idx_proj=_uni(g, (gen.HIDDEN, gen.IDX_HEADS), -1, 1),
                 hadamard_q=_uni(g, (gen.IDX_DIM, gen.IDX_DIM), -1, 1), hadamard_k=_uni(g, (gen.IDX_DIM, gen.IDX_DIM), -1, 1))
    else:
        w.update(w_uqqr=_uni(g, (gen.Q_LORA, up), -0.1, 0.1), w_idx_qb=_uni(g, (gen.Q_LORA, idx), -0.1, 0.1),
                 w_idx_k=_uni(g, (gen.HIDDEN, gen.IDX_DIM), -0.1, 0.1),
                 w_idx_proj=_uni(g, (gen.HIDDEN, gen.IDX_HEADS), -0.1, 0.1))
    return w


def _prolog_pages(case):
    """Every sequence's new tokens lie at the end of its pages; the prolog touches no other rows."""
    return [max(300, case["s1"]) + 7 * i % 90 for i in range(case["b"])]


def _prepare_prolog(case, seed):
    g = _gen(seed)
    b, s1 = case["b"], case["s1"]
    t = b * s1
    lens = _prolog_pages(case)
    block_num, _, table = gen.make_block_table(lens, g, "cuda")
    rows = block_num * 128
    w = _prolog_weights(g, True)
    x = _uni(g, (t, gen.HIDDEN), -1, 1)
    cos, sin = _uni(g, (t, 64), -0.1, 0.1), _uni(g, (t, 64), -0.1, 0.1)
    kv, kr = _int8(g, (rows, 512)), _uni(g, (rows, 64), -1, 1)
    ks = _uni(g, (rows, 4), 1e-3, 1e-2, torch.float32)
    ik, iks = _int8(g, (rows, 128)), _uni(g, (rows, 1), 1e-3, 1e-2, torch.float16)
    out = dict(
        q_nope=torch.zeros((t, 128, 512), dtype=BF16, device="cuda"), q_rope=torch.zeros((t, 128, 64), dtype=BF16, device="cuda"),
        q_int8=torch.zeros((t, 64, 128), dtype=torch.int8, device="cuda"),
        q_scale=torch.zeros((t, 64, 1), dtype=torch.float16, device="cuda"),
        weights=torch.zeros((t, 64), dtype=torch.float16, device="cuda"),
        kv=kv, kr=kr, kv_scales=ks, idx_k=ik, idx_k_scale=iks)
    op = pto.mla_indexer_prolog_quant_d if s1 <= 4 else pto.mla_indexer_prolog_quant_p
    call = _call(case, op, x, w["w_dq"], w["w_uqqr"], w["w_qb_scale"], w["w_uk"], w["w_dkvkr"], w["gamma_cq"],
                 w["gamma_ckv"], cos, sin, _new_rows(b, s1, lens, table), kv, kr, ks, w["w_idx_qb"], w["w_idx_qb_scale"],
                 w["w_idx_k"], w["w_idx_proj"], w["ln_gamma"], w["ln_beta"], w["hadamard_q"], w["hadamard_k"], ik, iks,
                 out["q_nope"], out["q_rope"], kv, kr, ks, out["q_int8"], out["q_scale"], ik, iks, out["weights"],
                 1e-5, 1e-5, "PA_BSND")
    return dict(call=call, out=out, keep=w)


def _prepare_layer(case, seed):
    g = _gen(seed)
    b, s1 = case["b"], case["s1"]
    t = b * s1
    lens = [max(s, s1) for s in _lengths(case)]
    block_num, _, table = gen.make_block_table(lens, g, "cuda")
    w = _prolog_weights(g, False)
    x = _uni(g, (b, s1, gen.HIDDEN), -1, 1)
    cos, sin = _uni(g, (b, s1, 64), -1, 1), _uni(g, (b, s1, 64), -1, 1)
    kv = _uni(g, (block_num, 128, 1, 512), -1, 1)
    kr, ik = _uni(g, (block_num, 128, 1, 64), -1, 1), _uni(g, (block_num, 128, 1, 128), -1, 1)
    act = torch.tensor(lens, dtype=torch.int32, device="cuda")
    att = torch.zeros((b, s1, 128, 512), dtype=BF16, device="cuda")
    scratch = dict(query_nope=torch.zeros((t, 128, 512), dtype=BF16, device="cuda"),
                   query_rope=torch.zeros((t, 128, 64), dtype=BF16, device="cuda"),
                   idx_query=torch.zeros((t, 64, 128), dtype=BF16, device="cuda"),
                   idx_weights=torch.zeros((t, 64), dtype=BF16, device="cuda"),
                   topk_res=torch.zeros((t, 1, TOPK), dtype=torch.int32, device="cuda"))
    call = _call(case, pto.decode_indexer_attention_layer, x, w["w_dq"], w["w_uqqr"], w["w_uk"], w["w_dkvkr"],
                 w["gamma_cq"], w["gamma_ckv"], sin, cos, _new_rows(b, s1, lens, table).reshape(b, s1), kv, kr, table, act,
                 w["w_idx_qb"], w["w_idx_k"], w["w_idx_proj"], w["ln_gamma"], w["ln_beta"], ik, att, scratch=scratch)
    out = {k: v for k, v in scratch.items() if k != "topk_res"}  # a set in no order, as in the fused chain
    out.update(attention=att, kv=kv, kr=kr, idx_k=ik)
    return dict(call=call, out=out, keep=w)


def prepare(case, seed):
    return {"decode": _prepare_decode, "indexer": _prepare_indexer, "attention": _prepare_attention,
            "prolog": _prepare_prolog, "layer": _prepare_layer}[case["op"]](case, seed)


def run(state):
    state["call"]()
    return state["out"]


# --- what a pass cannot do without --------------------------------------------------------------


def _indexer_work(lens, s1, key_bytes, query_bytes):
    """Keys (and their scales), queries, scales and weights once; the score product of every causal (query, key)."""
    b = f = 0
    for s in lens:
        b += s * key_bytes + s1 * query_bytes + 4 * math.ceil(s / 128) + s1 * TOPK * 4
        f += sum(2 * 64 * 128 * max(s - (s1 - 1 - i), 0) for i in range(s1))
    return b, f


def _attention_work(lens, s1, heads, row_bytes):
    """Selected rows (no more than the sequence has), queries, indices and output once; q.k over 576 and p.v over 512."""
    b = f = 0
    for s in lens:
        n = [min(max(s - (s1 - 1 - i), 0), TOPK) for i in range(s1)]
        b += min(sum(n), s) * row_bytes + sum(4 * v for v in n) + s1 * heads * (576 + 512) * 2
        f += sum(2 * heads * v * (576 + 512) for v in n)
    return b, f


def _prolog_work(t, quant):
    h, r, up, idx = gen.HIDDEN, gen.Q_LORA, 128 * 192, 64 * 128
    w = 1 if quant else 2
    b = 2 * h * (r + 576 + 192) + w * r * (up + idx) + 2 * 128 * 128 * 512
    b += (4 * (up + idx) + 2 * 2 * 128 * 128) if quant else 0
    token = 2 * h + 2 * 2 * 64 + 8 + 2 * 128 * (512 + 64)
    token += (64 * 128 + 2 * 64 + 2 * 64 + 512 + 128 + 16 + 128 + 2) if quant else (2 * 64 * 128 + 2 * 64 + 2 * (512 + 64 + 128))
    f = 2 * t * (h * (r + 576 + 192) + r * (up + idx) + 128 * 128 * 512) + (2 * t * 65 * 128 * 128 if quant else 0)
    return b + t * token, f


def work(case):
    op, s1 = case["op"], case["s1"]
    if op == "prolog":
        b, f = _prolog_work(case["b"] * s1, True)
        return {"bytes": b, "flops": f}
    lens = _lengths(case)
    scale = 2 if case.get("scales") == "f16" else 4
    b = f = 0
    if op in ("decode", "indexer"):
        b, f = _indexer_work(lens, s1, 128 + scale, 64 * 128 + 2 * 64 * scale)
    if op == "layer":
        lens = [max(s, s1) for s in lens]
        p = _prolog_work(case["b"] * s1, False)
        i = _indexer_work(lens, s1, 256, 64 * 128 * 2 + 64 * 2)
        b, f = p[0] + i[0], p[1] + i[1]
    if op in ("decode", "attention", "layer"):
        bf16 = op == "layer" or case.get("layout") == "bf16"
        a = _attention_work(lens, s1, case.get("heads", 128), 1152 if bf16 else gen.PACKED_ROW_BYTES)
        b, f = b + a[0], f + a[1]
    return {"bytes": b, "flops": f}


def tolerance(case):
    if case["op"] == "indexer":
        # positions in order of an fp32 sum of 64 terms: neighbours whose sums differ in the last bit may change places
        return {"rel": 0.0, "differ": 5e-3}
    # bf16 results of bf16 products: the order of the sums and the rounding of the unnormalised probabilities. int8 results
    # of the prolog: values whose bf16 or fp32 predecessor lies on a rounding boundary
    return {"rel": 1e-2, "differ": 5e-3}
