"""Sparse MLA attention on the GPU against the CPU oracle and the reference-made fixtures.
Tolerance (stated by the benchmark): max-abs 2e-2 and relative L2 5e-3 on the bf16 output."""
import pytest
import torch

import oracle
import pypto_b200 as pto
from pypto_b200 import _lib
from pypto_b200 import inputs as gen
from golden_util import SFA_CASES, from_np_bf16, load_case, mask_empty_rows

pytestmark = pytest.mark.gpu
DEV = "cuda"
MAX_ABS, REL_L2 = 2e-2, 5e-3
SCALE = 576 ** -0.5


def _run(d, packed=False, prefill=False, nq=128, bf16_cache=False):
    g = d.to(DEV)
    if bf16_cache:  # the non-quantised branch: the cache holds the values the int8 rows dequantise to
        g.key_nope_2d = oracle.dequantised_cache(d.key_nope_2d, d.k_nope_scales).to(DEV)
        g.k_nope_scales = torch.zeros(1, 4, device=DEV)  # not read
    out = torch.full((d.b, d.s1, nq, 512), 7.0, dtype=torch.bfloat16, device=DEV)
    cfg = pto.SaTileShapeConfig()
    if packed:
        cache = gen.pack_kv_rows(g.key_nope_2d, g.key_rope_2d, g.k_nope_scales)
        fn = pto.sparse_attention_antiquant_p if prefill else pto.sparse_attention_antiquant_d
        fn(g.query_nope, g.query_rope, cache, g.topk_indices, g.block_table, g.act_seq_key, out.reshape(-1, 512), nq,
           1, SCALE, 2048, 128, d.max_blocks, cfg)
    else:
        fn = pto.sparse_flash_attention_quant_p if prefill else pto.sparse_flash_attention_quant_d
        fn(pto.from_torch(g.query_nope, dynamic_axis=[0], name="q_nope"), g.query_rope, g.key_nope_2d, g.key_rope_2d,
           g.k_nope_scales, g.topk_indices, g.block_table, g.act_seq_key, out, nq, 1, SCALE, 2048, 128, d.max_blocks,
           cfg)
    torch.cuda.synchronize()
    assert pto.workspace_status()[0] == 0
    return out.cpu()


def _check(got, want):
    e = oracle.attention_errors(got, want)
    assert e["max_abs"] <= MAX_ABS and e["rel_l2"] <= REL_L2, e
    return e


@pytest.mark.parametrize("name", SFA_CASES)
@pytest.mark.parametrize("packed", [False, True], ids=["split_arrays", "packed_rows"])
def test_matches_reference_fixture(name, packed):
    d, z = load_case(name)
    want = mask_empty_rows(from_np_bf16(z["out_no_flash"]).reshape(d.b, d.s1, 128, 512), d)
    got = _run(d, packed=packed)
    _check(got, want)
    # per token too, so that a short row cannot hide behind a long one
    for bi in range(d.b):
        for i in range(d.s1):
            if d.act_seq[bi] - d.s1 + 1 + i > 0:
                _check(got[bi, i], want[bi, i])
            else:
                assert torch.all(got[bi, i] == 0)


def test_config0_against_oracle():
    """Benchmark configuration 0: batch 2, context 8192, 2048 selected rows, split over many CTAs."""
    d = gen.make_config(0)
    want = oracle.sparse_attention(d.query_nope, d.query_rope, d.key_nope_2d, d.key_rope_2d, d.k_nope_scales,
                                   d.topk_indices, d.block_table, d.act_seq, d.s1)
    e = _check(_run(d), want)
    print("config0 errors", e)


def test_many_tokens_unsplit_and_prefill_entry():
    """More than 148 (token, head-block) CTAs: the unsplit path that writes bf16 directly."""
    g = torch.Generator().manual_seed(8)
    act = torch.randint(1, 700, (40,), generator=g).tolist()
    d = gen.make_inputs(act, s1=2, seed=21, with_indexer=False, with_topk=True)
    want = oracle.sparse_attention(d.query_nope, d.query_rope, d.key_nope_2d, d.key_rope_2d, d.k_nope_scales,
                                   d.topk_indices, d.block_table, d.act_seq, d.s1)
    got = _run(d, prefill=True)
    _check(got, want)
    for bi in range(d.b):
        for i in range(d.s1):
            if act[bi] - 2 + 1 + i > 0:
                _check(got[bi, i], want[bi, i])
            else:
                assert torch.all(got[bi, i] == 0)


def test_head_slice_of_16():
    """16 heads per device, the head-sharded prefill layout."""
    d = gen.make_inputs([3000, 150], s1=1, seed=33, with_indexer=False, with_topk=True, attn_heads=16)
    want = oracle.sparse_attention(d.query_nope, d.query_rope, d.key_nope_2d, d.key_rope_2d, d.k_nope_scales,
                                   d.topk_indices, d.block_table, d.act_seq, d.s1, nq=16)
    _check(_run(d, nq=16), want)


@pytest.mark.parametrize("packed", [False, True], ids=["split_arrays", "packed_rows"])
@pytest.mark.parametrize("nq,lens,s1", [
    (16, [1, 127, 128, 129, 256, 257, 2048, 2500], 1),
    (16, [1, 79, 80, 81, 160, 161, 2048, 2500], 1),    # edges of its 80-row tiles; one item per SM and split
    (32, [63, 64, 65, 128, 2047, 130, 0, 3000], 2),    # edges of its 64-row tiles, tokens that see nothing
    (48, [700, 2100], 2),                              # three blocks of 16 heads
    (64, [300] * 90, 1),                               # more items than SMs: CTAs walk several, unsplit
])
def test_head_slices_at_tile_edges(nq, lens, s1, packed):
    d = gen.make_inputs(lens, s1=s1, seed=37 + nq, with_indexer=False, with_topk=True, attn_heads=nq)
    want = oracle.sparse_attention(d.query_nope, d.query_rope, d.key_nope_2d, d.key_rope_2d, d.k_nope_scales,
                                   d.topk_indices, d.block_table, d.act_seq, d.s1, nq=nq)
    got = _run(d, nq=nq, packed=packed)
    for bi in range(d.b):
        for i in range(d.s1):
            if d.act_seq[bi] - d.s1 + 1 + i > 0:
                _check(got[bi, i], want[bi, i])
            else:
                assert torch.all(got[bi, i] == 0)


def _uneven_inputs(kind, nq, act, s1):
    """Attention inputs whose terms differ much in size; the rest of a token's rows share an offset of their latent values,
    so that weight that is lost shows in the output."""
    d = gen.make_inputs(act, s1=s1, seed=71, with_indexer=False, with_topk=True, attn_heads=nq)
    g = torch.Generator().manual_seed(nq)
    offset = torch.randint(-60, 61, (1, 512), generator=g)
    d.key_nope_2d = (offset + torch.randint(-40, 41, d.key_nope_2d.shape, generator=g)).to(torch.int8)
    d.query_rope[:, :2] = 8.0
    d.key_rope_2d[:, :2] = 0.0
    for bi in range(d.b):
        table = d.block_table[bi].long()
        if kind.startswith("sink"):  # the sequence's first row, `nats` above the others; a token selects it first of all
            row = table[0] * 128
            nats = float(kind[4:])
            d.key_rope_2d[row, 0] = nats * 24.0 / 8.0
            d.key_nope_2d[row] = torch.randint(-3, 4, (512,), generator=g).to(torch.int8)
            for ti in range(bi * s1, (bi + 1) * s1):
                sel = d.topk_indices[ti]
                sel[(sel == 0).nonzero()] = sel[0].clone()
                sel[0] = 0
        elif kind == "scale":  # a row in 128 with a scale 300 times its neighbours', little weight and few values
            rows = table[torch.arange(act[bi] // 128)] * 128 + torch.randint(0, 128, (act[bi] // 128,), generator=g)
            d.k_nope_scales[rows] = 1.5
            d.key_rope_2d[rows, 1] = -9.0
            d.key_nope_2d[rows] = (torch.rand((rows.numel(), 512), generator=g) < 0.02).to(torch.int8)
    if kind == "query":  # one dim of every query a hundred times the others
        d.query_nope[:, 5] *= 100.0
    return d


@pytest.mark.parametrize("nq", [16, 64, 128])
@pytest.mark.parametrize("act,s1", [([2300, 700], 2), ([2400], 148)], ids=["split", "unsplit"])
@pytest.mark.parametrize("kind", ["sink7", "sink9", "sink11", "scale", "query"])
def test_terms_of_very_different_size(kind, act, s1, nq):
    """Against 64 bits, per token and head, since a norm over the whole output hides single heads. The bound: probabilities (or
    probability times row scale), row values and outputs are rounded to bf16 once each, 2^-9 of a term at most. The dominant
    term may meet the worst of the first two; the other terms' and the output's roundings are independent (0.0011 rms):
    2 * 2^-9 + 0.0011 = REL_L2. (The oracle rounds its probabilities to bf16 as well: up to another 2^-9 apart.)"""
    s1 = s1 if nq == 16 or s1 == 2 else 80
    d = _uneven_inputs(kind, nq, act, s1)
    got = _run(d, nq=nq).double()
    for ti in range(d.t):
        bi, i = divmod(ti, s1)
        sel = d.topk_indices[ti, :min(act[bi] - s1 + 1 + i, 2048)].long()
        rows = d.block_table[bi].long()[sel // 128] * 128 + sel % 128
        v = (d.key_nope_2d[rows].double().reshape(-1, 4, 128) * d.k_nope_scales[rows].double()[:, :, None]).reshape(-1, 512)
        qn, qr = (q.reshape(d.t, nq, -1)[ti].double() for q in (d.query_nope, d.query_rope))
        want = torch.softmax((qn @ v.T + qr @ d.key_rope_2d[rows].double().T) * SCALE, dim=-1) @ v
        err = (got[bi, i] - want).norm(dim=-1) / want.norm(dim=-1)
        assert float(err.max()) <= REL_L2, (ti, float(err.max()), float(err.mean()))


@pytest.mark.parametrize("tokens", [1, 14, 15, 24, 37], ids=lambda t: f"{t}_tokens")  # 16, 5, 4, 3 and 2 splits
def test_merge_of_splits(tokens):
    d = gen.make_inputs([(1, 130, 300, 700)[i % 4] for i in range(tokens)], s1=1, seed=tokens, with_indexer=False, with_topk=True)
    want = oracle.sparse_attention(d.query_nope, d.query_rope, d.key_nope_2d, d.key_rope_2d, d.k_nope_scales,
                                   d.topk_indices, d.block_table, d.act_seq, d.s1)
    _check(_run(d), want)


@pytest.mark.parametrize("tokens", [74, 75, 111, 112, 149], ids=lambda t: f"{t}_tokens")  # rests of 0, 1, 37, 38 and 1: 1, 16, 2, 1 and 16 splits
@pytest.mark.parametrize("longest", [700, 1500])  # rows of few tiles are not split behind a whole round
def test_split_of_the_last_round(tokens, longest):
    act = [(1, 130, 300, 5)[i % 4] for i in range(tokens)]
    act[0] = act[73] = act[-1] = longest
    d = gen.make_inputs(act, s1=1, seed=tokens, with_indexer=False, with_topk=True)
    want = oracle.sparse_attention(d.query_nope, d.query_rope, d.key_nope_2d, d.key_rope_2d, d.k_nope_scales,
                                   d.topk_indices, d.block_table, d.act_seq, d.s1)
    _check(_run(d), want)
    assert torch.equal(_run(d, bf16_cache=True), _run(d))


def test_a_workspace_without_room_for_the_last_round():
    """A C caller's workspace of the size that the call needs and no more: the same call, unsplit."""
    d = gen.make_inputs([1500] + [130] * 73 + [1500], s1=1, seed=6, with_indexer=False, with_topk=True)
    want = _run(d)
    g, lib = d.to(DEV), _lib.load()
    assert lib.pto_sfa_extra_bytes(75, 128) > 0
    ws = torch.zeros(lib.pto_sfa_workspace_bytes(75, 128), dtype=torch.uint8, device=DEV)
    out = torch.zeros((75, 1, 128, 512), dtype=torch.bfloat16, device=DEV)
    rc = lib.pto_sfa_quant(*(x.data_ptr() for x in (g.query_nope, g.query_rope, g.key_nope_2d, g.key_rope_2d, g.k_nope_scales,
                                                    g.topk_indices, g.block_table, g.act_seq_key, out)),
                           75, 1, 128, 1, SCALE, 2048, 128, g.key_nope_2d.shape[0], d.max_blocks, 128, 0, ws.data_ptr(), ws.numel(),
                           torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0 and int(ws[:4].view(torch.int32)) == 0
    _check(out.cpu(), want)
    assert torch.equal(out.cpu()[1:74], want[1:74])


@pytest.mark.parametrize("nq", [128, 16])
@pytest.mark.parametrize("block_size", [1, 2, 3, 100, 4096])  # the kernels divide a position by it through a reciprocal
def test_block_sizes_address_the_same_rows(block_size, nq):
    n = 1201
    d = gen.make_inputs([n], s1=1, seed=5, with_indexer=False, with_topk=True, attn_heads=nq)
    rows = d.block_table[0].long()[torch.arange(n) // 128] * 128 + torch.arange(n) % 128  # row of each position
    pages = -(-n // block_size)
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(block_size))    # where each page of the new cache lies
    place = order[torch.arange(n) // block_size] * block_size + torch.arange(n) % block_size
    total = pages * block_size
    kn, kr, ks = (torch.zeros(total, x.shape[1], dtype=x.dtype) for x in (d.key_nope_2d, d.key_rope_2d, d.k_nope_scales))
    for dst, src in ((kn, d.key_nope_2d), (kr, d.key_rope_2d), (ks, d.k_nope_scales)):
        dst[place] = src[rows]
    out = torch.zeros((1, 1, nq, 512), dtype=torch.bfloat16, device=DEV)
    pto.sparse_flash_attention_quant_d(d.query_nope.to(DEV), d.query_rope.to(DEV), kn.to(DEV), kr.to(DEV), ks.to(DEV),
                                       d.topk_indices.to(DEV), order.to(torch.int32)[None].contiguous().to(DEV),
                                       d.act_seq_key.to(DEV), out, nq, 1, SCALE, 2048, block_size, pages)
    torch.cuda.synchronize()
    assert pto.workspace_status()[0] == 0
    assert torch.equal(out.cpu(), _run(d, nq=nq))


@pytest.mark.parametrize("nq", [128, 16, 32])
def test_latent_cache_on_a_16_byte_boundary(nq):
    """32-byte loads take caches on a 32-byte boundary, 16-byte ones any other: the same values either way."""
    d = gen.make_inputs([3000, 700], s1=1, seed=8, with_indexer=False, with_topk=True, attn_heads=nq)
    want = _run(d, nq=nq)
    g = d.to(DEV)
    raw = torch.zeros(g.key_nope_2d.numel() + 48, dtype=torch.int8, device=DEV)
    at = -raw.data_ptr() % 32 + 16
    kn = raw[at:at + g.key_nope_2d.numel()].view(-1, 512)
    kn.copy_(g.key_nope_2d)
    assert kn.data_ptr() % 32 == 16
    out = torch.zeros((d.b, 1, nq, 512), dtype=torch.bfloat16, device=DEV)
    pto.sparse_flash_attention_quant_d(g.query_nope, g.query_rope, kn, g.key_rope_2d, g.k_nope_scales, g.topk_indices, g.block_table,
                                       g.act_seq_key, out, nq, 1, SCALE, 2048, 128, d.max_blocks)
    torch.cuda.synchronize()
    assert pto.workspace_status()[0] == 0
    assert torch.equal(out.cpu(), want)


@pytest.mark.parametrize("tokens", [16, 17, 74, 75])  # from 17 to 74 read in 16-byte loads wherever the cache lies, if the longest has
@pytest.mark.parametrize("longest", [700, 4224])       # more than 4096 keys
def test_latent_cache_on_a_16_byte_boundary_over_token_counts(tokens, longest):
    act = [(700, 130, 1, 5)[i % 4] for i in range(tokens)]
    act[1] = longest
    d = gen.make_inputs(act, s1=1, seed=tokens, with_indexer=False, with_topk=True)
    want = _run(d)
    _check(want, oracle.sparse_attention(d.query_nope, d.query_rope, d.key_nope_2d, d.key_rope_2d, d.k_nope_scales, d.topk_indices,
                                         d.block_table, d.act_seq, d.s1))
    g = d.to(DEV)
    raw = torch.zeros(g.key_nope_2d.numel() + 48, dtype=torch.int8, device=DEV)
    at = -raw.data_ptr() % 32 + 16
    kn = raw[at:at + g.key_nope_2d.numel()].view(-1, 512)
    kn.copy_(g.key_nope_2d)
    out = torch.zeros((tokens, 1, 128, 512), dtype=torch.bfloat16, device=DEV)
    pto.sparse_flash_attention_quant_d(g.query_nope, g.query_rope, kn, g.key_rope_2d, g.k_nope_scales, g.topk_indices, g.block_table,
                                       g.act_seq_key, out, 128, 1, SCALE, 2048, 128, d.max_blocks)
    torch.cuda.synchronize()
    assert pto.workspace_status()[0] == 0
    assert torch.equal(out.cpu(), want)


def test_order_of_indices_does_not_matter_beyond_rounding():
    d = gen.make_inputs([5000], s1=1, seed=2, with_indexer=False, with_topk=True)
    a = _run(d)
    d.topk_indices = d.topk_indices.flip(-1).contiguous()
    b = _run(d)
    _check(a, b)


@pytest.mark.parametrize("name", SFA_CASES)
def test_bf16_cache_matches_reference_fixture(name):
    """Non-quantised `key_nope_2d` (the golden's is_kn_quant = 0): the reference's output over the bf16
    cache of dequantised values is the fixture's `out_no_flash` itself."""
    d, z = load_case(name)
    assert bool(z["out_bf16_equals_no_flash"])
    want = mask_empty_rows(from_np_bf16(z["out_no_flash"]).reshape(d.b, d.s1, 128, 512), d)
    got = _run(d, bf16_cache=True)
    _check(got, want)
    for bi in range(d.b):
        for i in range(d.s1):
            if d.act_seq[bi] - d.s1 + 1 + i > 0:
                _check(got[bi, i], want[bi, i])
            else:
                assert torch.all(got[bi, i] == 0)
    # the key tiles hold the values the int8 path dequantises to and both caches run the same kernel (only the
    # producers differ): the outputs are equal bit for bit
    assert torch.equal(got, _run(d))


def test_bf16_cache_many_tokens_and_split():
    """Both launch shapes of the bf16 branch: config 0 (2 tokens, split over CTAs) and 80 ragged tokens."""
    d = gen.make_config(0)
    assert torch.equal(_run(d, bf16_cache=True), _run(d))
    g = torch.Generator().manual_seed(18)
    act = torch.randint(1, 900, (40,), generator=g).tolist()
    d = gen.make_inputs(act, s1=2, seed=23, with_indexer=False, with_topk=True)
    want = oracle.sparse_attention(d.query_nope, d.query_rope, oracle.dequantised_cache(d.key_nope_2d, d.k_nope_scales),
                                   d.key_rope_2d, None, d.topk_indices, d.block_table, d.act_seq, d.s1)
    got = _run(d, bf16_cache=True, prefill=True)
    _check(got, want)
    assert torch.equal(got, _run(d))


def test_bf16_cache_head_slice_is_refused():
    d = gen.make_inputs([300], s1=1, seed=3, with_indexer=False, with_topk=True, attn_heads=16)
    with pytest.raises(RuntimeError, match="128 heads"):
        _run(d, nq=16, bf16_cache=True)


@pytest.mark.parametrize("name", SFA_CASES)
def test_packed_rows_equal_split_arrays_bit_for_bit(name):
    """The packed 656-byte rows and the three split arrays hold the same bytes and go through the same kernel."""
    d, _ = load_case(name)
    assert torch.equal(_run(d, packed=True), _run(d, packed=False))
