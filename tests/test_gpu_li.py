"""Lightning indexer on the GPU against the CPU oracle and the reference-made fixtures.
Everything goes through the operator wrappers, i.e. through the C ABI."""
import pytest
import torch

import oracle
import pypto_b200 as pto
from pypto_b200 import _lib
from pypto_b200 import inputs as gen
from golden_util import LI_CASES, load_case

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _scores(d, simt, first_mm=False):
    g = d.to(DEV)
    stride = d.max_blocks * 128
    sc = torch.full((d.t, stride), float("nan"), dtype=torch.float32, device=DEV)
    fm = torch.zeros((d.t * 64, stride), dtype=torch.float16, device=DEV) if first_mm else None
    pto.lightning_indexer_scores(g.idx_query, g.idx_query_scale, g.idx_key_cache, g.idx_key_scale, g.idx_weight,
                                 g.act_seq_key, g.block_table, sc, fm, simt=simt)
    torch.cuda.synchronize()
    return sc.cpu(), (fm.cpu() if fm is not None else None)


def _decode(d, **kw):
    g = d.to(DEV)
    out = torch.zeros((d.t, 1, 2048), dtype=torch.int32, device=DEV)
    pto.lightning_indexer_decode(pto.from_torch(g.idx_query, name="idx_query", dynamic_axis=[0]), g.idx_query_scale,
                                 g.idx_key_cache, g.idx_key_scale, g.idx_weight, g.act_seq_key, g.block_table,
                                 pto.from_torch(out), [128, 64, 32, 16, 8, 4, 1], pto.LightningIndexerConfigs(), 2048,
                                 **kw)
    torch.cuda.synchronize()
    assert pto.workspace_status()[0] == 0
    return out.cpu()


def _check_rows(sc, rows, d, rtol):
    for ti, row in enumerate(rows):
        n = row.numel()
        torch.testing.assert_close(sc[ti, :n], row, rtol=rtol, atol=1e-9)
        # positions past the sequence are left untouched
        assert torch.isnan(sc[ti, n:]).all()


@pytest.mark.parametrize("name", LI_CASES)
@pytest.mark.parametrize("simt", [True, False], ids=["simt", "tcgen05"])
def test_scores_match_oracle_on_fixtures(name, simt):
    d, z = load_case(name)
    rows, first_mm = oracle.li_oracle.li_scores(d.idx_query, d.idx_query_scale, d.idx_key_cache, d.idx_key_scale,
                                                d.idx_weight, d.act_seq, d.block_table, d.s1, return_first_mm=True)
    sc, fm = _scores(d, simt, first_mm=simt)
    # same formula; the 64-term fp32 head sum is taken in a different order
    _check_rows(sc, rows, d, rtol=3e-6)
    mm_out = torch.from_numpy(z["mm_out"])
    for ti, row in enumerate(rows):
        torch.testing.assert_close(sc[ti, :row.numel()], mm_out[ti, :row.numel()], rtol=3e-6, atol=1e-9)
    if simt:
        for ti, row in enumerate(rows):  # fp16 relu(dot)/2048 tiles: bit-exact
            assert torch.equal(fm[ti * 64:(ti + 1) * 64, :row.numel()], first_mm[ti])


@pytest.mark.parametrize("s1", [1, 2, 3, 4])
def test_integer_dots_bit_exact(s1):
    """One-hot head weight with unit scales turns the score into fp16(relu(q_h.k)/2048) itself,
    which exposes every int32 dot product of the tensor-core path exactly."""
    act = [1000, 77, 513][: max(1, 4 - s1)] + [300]
    d = gen.make_inputs(act, s1=s1, seed=11 + s1, with_attention=False)
    d.idx_query_scale.fill_(1.0)
    d.idx_key_scale.fill_(1.0)
    for head in (0, 21, 63):
        d.idx_weight.zero_()
        d.idx_weight[:, head] = 1.0
        rows, first_mm = oracle.li_oracle.li_scores(d.idx_query, d.idx_query_scale, d.idx_key_cache, d.idx_key_scale,
                                                    d.idx_weight, d.act_seq, d.block_table, d.s1, return_first_mm=True)
        sc, _ = _scores(d, simt=False)
        for ti, row in enumerate(rows):
            want = first_mm[ti][head].to(torch.float32)
            assert torch.equal(sc[ti, :row.numel()], want), f"token {ti} head {head}"
            assert torch.equal(row, want)


def test_tensor_core_scores_equal_simt_scores_on_large_ragged_batch():
    g = torch.Generator().manual_seed(5)
    act = torch.randint(1, 9000, (37,), generator=g).tolist() + [16384, 128, 127, 129]
    d = gen.make_inputs(act, s1=2, seed=99, scale_dtype=torch.float16, with_attention=False)
    a, _ = _scores(d, simt=True)
    b, _ = _scores(d, simt=False)
    for bi, s in enumerate(act):
        for i in range(2):
            torch.testing.assert_close(b[bi * 2 + i, :s], a[bi * 2 + i, :s], rtol=3e-6, atol=1e-9)
    assert pto.workspace_status()[0] == 0


@pytest.mark.parametrize("name", LI_CASES)
@pytest.mark.parametrize("simt", [True, False], ids=["simt", "tcgen05"])
def test_topk_matches_reference_fixture(name, simt):
    d, z = load_case(name)
    got = _decode(d, _simt_scores=simt)
    want = torch.from_numpy(z["topk_res"])
    mm_out = torch.from_numpy(z["mm_out"])
    for ti in range(d.t):
        untied, tied = oracle.topk_set_diff(got[ti], want[ti], mm_out[ti])
        assert untied == 0, f"row {ti}: {untied} untied differences ({tied} tied)"
        bi, i = divmod(ti, d.s1)
        eff = max(0, min(2048, d.act_seq[bi] - (d.s1 - 1 - i)))
        assert torch.all(got[ti, 0, :eff] >= 0) and torch.all(got[ti, 0, eff:] == -1)
        assert len(set(got[ti, 0, :eff].tolist())) == eff
        # value-descending order
        vals = mm_out[ti][got[ti, 0, :eff].long()]
        assert torch.all(vals[:-1] >= vals[1:] - 1e-6 * vals[:-1].abs())


def test_topk_stage_exact_on_kernel_scores():
    """Selection alone: over the kernel's own score rows the selected set must equal torch.topk's
    exactly (ties broken toward the smaller position)."""
    g = torch.Generator().manual_seed(3)
    rows = [5000, 2049, 2048, 131072, 40000, 1, 70000]
    stride = 131072
    sc = torch.randn((len(rows), stride), generator=g)
    sc[4, :40000] = torch.randint(0, 50, (40000,), generator=g).float()  # heavy ties
    sc[6, :70000] = 1.25  # all equal: the radix path must pick the 2048 smallest positions
    act = torch.tensor(rows, dtype=torch.int32)
    out = torch.zeros((len(rows), 1, 2048), dtype=torch.int32, device=DEV)
    pto.lightning_indexer_topk(sc.to(DEV), act.to(DEV), out, s1=1, selected_count=2048)
    torch.cuda.synchronize()
    out = out.cpu()
    for r, n in enumerate(rows):
        k = min(n, 2048)
        key = sc[r, :n].double() * 1e6 - torch.arange(n).double() * 1e-3 if r in (4, 6) else sc[r, :n].double()
        want = torch.topk(key, k).indices
        assert set(out[r, 0, :k].tolist()) == set(want.tolist()), f"row {r}"
        assert torch.all(out[r, 0, k:] == -1)
        # value-descending, ties toward the smaller position (rows this long are scanned by a cluster of CTAs)
        got_keys = key[out[r, 0, :k].long()]
        assert torch.all(got_keys[:-1] >= got_keys[1:]), f"row {r} not ordered"
    # unsorted variant selects the same sets
    out2 = torch.zeros_like(out, device=DEV)
    pto.lightning_indexer_topk(sc.to(DEV), act.to(DEV), out2, s1=1, selected_count=2048, sort=False)
    torch.cuda.synchronize()
    for r, n in enumerate(rows):
        assert set(out2[r, 0].cpu().tolist()) == set(out[r, 0].tolist())


def test_config1_shape_against_oracle():
    """Benchmark configuration 1 (batch 8, context 32768) end to end."""
    d = gen.make_config(1)
    idx, vals, rows = oracle.lightning_indexer(d.idx_query, d.idx_query_scale, d.idx_key_cache, d.idx_key_scale,
                                               d.idx_weight, d.act_seq, d.block_table, d.s1)
    got = _decode(d)
    for ti in range(d.t):
        untied, _ = oracle.topk_set_diff(got[ti], idx[ti], rows[ti])
        assert untied == 0


@pytest.mark.parametrize("simt", [False, True], ids=["tcgen05", "simt"])
def test_rejected_page_sets_status_without_fault(simt):
    d = gen.make_inputs([700, 300], s1=1, seed=4, with_attention=False)
    d.block_table[0, 2] = d.block_num + 5  # outside the cache: the page is skipped and reads as zeros
    pto.reset_workspace_status()
    g = d.to(DEV)
    out = torch.zeros((d.t, 1, 2048), dtype=torch.int32, device=DEV)
    pto.lightning_indexer_decode(g.idx_query, g.idx_query_scale, g.idx_key_cache, g.idx_key_scale, g.idx_weight,
                                 g.act_seq_key, g.block_table, out, None, None, 2048, _simt_scores=simt)
    st = pto.workspace_status()
    assert st[0] & 0x1 and st[1] == d.block_num + 5
    pto.reset_workspace_status()
    assert pto.workspace_status()[0] == 0
    # both score kernels give the rejected page's 128 positions the score 0, whatever the buffer held before
    sc = torch.full((d.t, d.max_blocks * 128), float("nan"), dtype=torch.float32, device=DEV)
    pto.lightning_indexer_scores(g.idx_query, g.idx_query_scale, g.idx_key_cache, g.idx_key_scale, g.idx_weight,
                                 g.act_seq_key, g.block_table, sc, simt=simt)
    torch.cuda.synchronize()
    assert torch.all(sc[0, 256:384] == 0) and not torch.isnan(sc[0, :700]).any()
    pto.reset_workspace_status()


@pytest.mark.parametrize("name", [n for n in LI_CASES if n.endswith("f16")])
@pytest.mark.parametrize("simt", [True, False], ids=["simt", "tcgen05"])
def test_fp16_chain_formulation_matches_st_golden(name, simt):
    """The older formulation (LightningIndexerTopkImpl, flag PTO_LI_FP16_CHAIN): scores against the ST golden's
    quantised branch (every fp16 step reproduces exactly; the fp32 head sum is taken in another order), selected
    sets exact on untied scores."""
    d, z = load_case(name)
    g = d.to(DEV)
    stride = d.max_blocks * 128
    sc = torch.full((d.t, stride), float("nan"), dtype=torch.float32, device=DEV)
    pto.lightning_indexer_scores(g.idx_query, g.idx_query_scale, g.idx_key_cache, g.idx_key_scale, g.idx_weight,
                                 g.act_seq_key, g.block_table, sc, None, simt=simt, fp16_chain=True)
    torch.cuda.synchronize()
    sc = sc.cpu()
    want_rows = torch.from_numpy(z["chain_rows"])
    rows = oracle.li_scores_fp16_chain(d.idx_query, d.idx_query_scale, d.idx_key_cache, d.idx_key_scale, d.idx_weight,
                                       d.act_seq, d.block_table, d.s1)
    for bi in range(d.b):
        for i in range(d.s1):
            ti = bi * d.s1 + i
            eff = d.act_seq[bi] - (d.s1 - 1 - i)
            torch.testing.assert_close(sc[ti, :d.act_seq[bi]], rows[ti], rtol=3e-6, atol=1e-9)
            if eff > 0:
                torch.testing.assert_close(sc[ti, :eff], want_rows[ti, :eff], rtol=3e-6, atol=1e-9)
    got = _decode(d, _simt_scores=simt, fp16_chain=True)
    want = torch.from_numpy(z["chain_topk_res"])
    for ti in range(d.t):
        untied, _ = oracle.topk_set_diff(got[ti], want[ti], want_rows[ti])
        assert untied == 0, f"row {ti}: {untied} untied differences"


def test_fp16_chain_needs_fp16_scales():
    d = gen.make_inputs([300], s1=1, seed=5, scale_dtype=torch.float32, with_attention=False)
    g = d.to(DEV)
    sc = torch.zeros((d.t, d.max_blocks * 128), dtype=torch.float32, device=DEV)
    with pytest.raises(RuntimeError, match="fp16"):
        pto.lightning_indexer_scores(g.idx_query, g.idx_query_scale, g.idx_key_cache, g.idx_key_scale, g.idx_weight,
                                     g.act_seq_key, g.block_table, sc, None, fp16_chain=True)


@pytest.mark.parametrize("s1", [1, 2, 3, 4])
@pytest.mark.parametrize("spread", [0, 12, 30])
def test_head_weights_of_very_different_size(s1, spread):
    """The head sum takes fp32 weights as limbs of a common scale (two and more query tokens): weights that span 2^spread,
    a token whose weights are all zero, and the CUDA-core kernel's fp32 sums as the reference."""
    d = gen.make_inputs([700, 130], s1=s1, seed=60 + s1)
    g = torch.Generator().manual_seed(spread)
    d.idx_weight = d.idx_weight * torch.pow(2.0, -torch.randint(0, spread + 1, d.idx_weight.shape, generator=g).float())
    d.idx_weight[-1] = 0
    got, want = _scores(d, False)[0], _scores(d, True)[0]
    for ti in range(d.t):
        n = d.act_seq[ti // s1]
        torch.testing.assert_close(got[ti, :n], want[ti, :n], rtol=3e-6, atol=float(want[ti, :n].abs().max()) * 1e-6)


@pytest.mark.parametrize("s1", [2, 4])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("spread", [0, 6, 12])
def test_head_sum_is_no_further_from_64_bits_than_an_fp32_sum(s1, dtype, spread):
    """The head sum on the tensor cores (two and more query tokens) against the fp32 sum on CUDA cores (one), over the same rows:
    root mean square error and mean error, relative to the sum of the terms' sizes."""
    d = gen.make_inputs([6000, 900], s1=s1, seed=80 + spread, with_attention=False, scale_dtype=dtype).to(DEV)
    g = torch.Generator(device=DEV).manual_seed(spread)
    small = torch.pow(2.0, -torch.randint(0, spread + 1, d.idx_weight.shape, generator=g, device=DEV).float())
    d.idx_weight = (d.idx_weight.float().abs() * small).to(dtype)

    def scores(act, table):
        sc = torch.zeros((d.t, d.max_blocks * 128), device=DEV)
        pto.lightning_indexer_scores(d.idx_query, d.idx_query_scale, d.idx_key_cache, d.idx_key_scale, d.idx_weight, act, table, sc)
        return sc.double()

    tc = scores(d.act_seq_key, d.block_table)
    fp32 = scores(d.act_seq_key.repeat_interleave(s1), d.block_table.repeat_interleave(s1, 0).contiguous())
    err = {"tc": [], "fp32": []}
    for ti in range(d.t):
        pos = torch.arange(d.act_seq[ti // s1], device=DEV)
        rows = d.block_table[ti // s1].long()[pos // 128] * 128 + pos % 128
        dots = torch.relu(d.idx_key_cache.reshape(-1, 128)[rows].double() @ d.idx_query[ti].double().T)
        h = (dots / 2048).to(torch.float16).double()
        want = (h @ (d.idx_query_scale[ti] * d.idx_weight[ti]).double()) * d.idx_key_scale.reshape(-1)[rows].double()
        for name, got in (("tc", tc), ("fp32", fp32)):
            err[name].append((got[ti, :pos.numel()] - want) / want.clamp(min=1e-30))
    tc_err, fp32_err = torch.cat(err["tc"]), torch.cat(err["fp32"])
    assert float(tc_err.square().mean().sqrt()) <= float(fp32_err.square().mean().sqrt())
    assert abs(float(tc_err.mean())) <= 2.0 ** -28  # no truncation towards zero (rounding alone: 2^-25 over the root of 13800)


@pytest.mark.parametrize("s1", [1, 2, 4])
def test_infinite_head_weights(s1):
    """A weight that overflowed decides the scores of the keys that its head sees, and only those, as in the CUDA-core sum."""
    d = gen.make_inputs([700, 600], s1=s1, seed=66, with_attention=False)
    d.idx_weight[0, 3] = float("inf")
    d.idx_weight[-1, 40] = float("-inf")
    got, want = _scores(d, False)[0], _scores(d, True)[0]
    for ti in range(d.t):
        a, b = (v[ti, :d.act_seq[ti // s1]] for v in (got, want))
        torch.testing.assert_close(a, b, rtol=3e-6, atol=float(b.nan_to_num(0, 0, 0).abs().max()) * 1e-6, equal_nan=True)
        assert bool(torch.isinf(a).any()) == (ti in (0, d.t - 1))


@pytest.mark.parametrize("s1", [3, 4])
def test_three_and_four_query_tokens_with_many_pages_per_cta(s1):
    """s1 = 3, 4 leave room for two accumulator slots only; with more than four pages per CTA every slot is
    reused many times by the epilogue warps (one sequence of 131072 keys: about seven pages per CTA). The
    tensor-core scores must equal the CUDA-core kernel's."""
    d = gen.make_inputs([131072], s1=s1, seed=60 + s1, with_attention=False)
    a, _ = _scores(d, simt=True)
    b, _ = _scores(d, simt=False)
    assert pto.workspace_status()[0] == 0
    for i in range(s1):
        torch.testing.assert_close(b[i, :131072], a[i, :131072], rtol=3e-6, atol=1e-9)


def test_prefill_chunk_groups_share_a_launch():
    """22 query tokens per sequence: five full groups of four go into one launch (grid y), the last two tokens
    into a second one. Scores equal the CUDA-core kernel's for every token."""
    d = gen.make_inputs([9000, 300], s1=22, seed=77, with_attention=False)
    a, _ = _scores(d, simt=True)
    b, _ = _scores(d, simt=False)
    assert pto.workspace_status()[0] == 0
    for bi, s in enumerate(d.act_seq):
        for i in range(22):
            torch.testing.assert_close(b[bi * 22 + i, :s], a[bi * 22 + i, :s], rtol=3e-6, atol=1e-9)


@pytest.mark.parametrize("kind", ["float32", "float16", "fp16_chain"])
@pytest.mark.parametrize("n,s1", [(40, 40), (1030, 1030), (2300, 131), (5000, 9), (20, 50), (1200, 1024)])
def test_pages_behind_the_causal_end_are_left_out(n, s1, kind):
    """A chunk of one prompt: the selection of the chained call equals the selection alone over whole score rows. Groups of four
    tokens that begin before, at and behind the ends of pages, tokens that see no key, a last group of its own."""
    d = gen.make_inputs([n], s1=s1, seed=n + s1, with_attention=False,
                        scale_dtype=torch.float32 if kind == "float32" else torch.float16)
    g = d.to(DEV)
    sc = torch.full((d.t, d.max_blocks * 128), float("nan"), dtype=torch.float32, device=DEV)
    pto.lightning_indexer_scores(g.idx_query, g.idx_query_scale, g.idx_key_cache, g.idx_key_scale, g.idx_weight, g.act_seq_key,
                                 g.block_table, sc, fp16_chain=kind == "fp16_chain")
    assert torch.isfinite(sc[:, :n]).all()
    want = torch.zeros((d.t, 1, 2048), dtype=torch.int32, device=DEV)
    pto.lightning_indexer_topk(sc, g.act_seq_key, want, s1, 2048)
    assert torch.equal(_decode(d, fp16_chain=kind == "fp16_chain").cpu(), want.cpu())


@pytest.mark.parametrize("s1", [1, 2, 3])
def test_chained_selection_from_the_score_kernels_histogram_equals_the_two_stages(s1):
    """Asked to (`histogram=True`), with at most two query tokens per sequence, the score kernel leaves a 4096-bin
    histogram per row and the selection starts from it (one scan of the row, a radix step over the candidates in
    shared memory); with three tokens it scans the row for min/max and its own histogram as it does by default.
    Either way the ordered result must equal the selection run alone over the same score rows. Cases: ragged
    lengths, sequences whose causal end cuts a page, a row shorter than k, and rows whose scores all tie (zero
    weights: one bin holds the whole row, which sends the selection back to its own passes and the radix path)."""
    g0 = torch.Generator().manual_seed(50 + s1)
    act = torch.randint(2049, 30000, (6,), generator=g0).tolist() + [2048 + s1, 300, 9000, 4097]
    d = gen.make_inputs(act, s1=s1, seed=91 + s1, with_attention=False)
    d.idx_weight[8 * s1:9 * s1] = 0  # sequence 8: every score is +0
    got = _decode(d, histogram=True)
    assert torch.equal(got, _decode(d))
    g = d.to(DEV)
    sc = torch.zeros((d.t, d.max_blocks * 128), dtype=torch.float32, device=DEV)
    pto.lightning_indexer_scores(g.idx_query, g.idx_query_scale, g.idx_key_cache, g.idx_key_scale, g.idx_weight,
                                 g.act_seq_key, g.block_table, sc)
    want = torch.zeros((d.t, 1, 2048), dtype=torch.int32, device=DEV)
    pto.lightning_indexer_topk(sc, g.act_seq_key, want, s1=s1, selected_count=2048)
    torch.cuda.synchronize()
    assert torch.equal(got, want.cpu())
    # the tied rows select the smallest positions
    for i in range(s1):
        assert got[8 * s1 + i, 0].tolist() == list(range(2048))
    # unordered output: the same sets
    got_u = _decode(d, sort=False, histogram=True)
    for ti in range(d.t):
        assert set(got_u[ti, 0].tolist()) == set(got[ti, 0].tolist())


def test_two_ctas_per_row_with_thousands_of_tied_candidates():
    """24 rows: two CTAs per row. Unordered output with a single exchange between them: rank 1 writes its selected
    positions from the end of the row and pushes its candidates to the end of rank 0's buffer. Rows of eight
    distinct values put ~3700 keys into the threshold bucket, half in each rank, so that the two candidate segments
    overlap when rank 0 joins them; rows of 300 distinct values are the ordinary case."""
    g = torch.Generator().manual_seed(11)
    n, rows = 30000, 24
    sc = torch.empty((rows, 32768))
    sc[:12, :n] = torch.randint(0, 8, (12, n), generator=g).float()
    sc[12:, :n] = torch.randint(0, 300, (12, n), generator=g).float()
    act = torch.full((rows,), n, dtype=torch.int32)
    out = torch.zeros((rows, 1, 2048), dtype=torch.int32, device=DEV)
    pto.lightning_indexer_topk(sc.to(DEV), act.to(DEV), out, s1=1, selected_count=2048, sort=False)
    torch.cuda.synchronize()
    assert pto.workspace_status()[0] == 0
    out = out.cpu()
    for r in range(rows):
        key = sc[r, :n].double() * 1e6 - torch.arange(n).double() * 1e-3  # ties toward the smaller position
        want = set(torch.topk(key, 2048).indices.tolist())
        got = out[r, 0].tolist()
        assert len(set(got)) == 2048 and set(got) == want, f"row {r}"


@pytest.mark.parametrize("sort", [True, False], ids=["ordered", "unordered"])
@pytest.mark.parametrize("rows,n,k", [
    (3, 2047, 2048), (3, 2049, 2048), (2, 6144, 2048), (2, 6145, 2048),   # rows that are the list, and the first that are not
    (5, 8192, 7), (2, 8193, 1), (40, 20000, 2048), (9, 32769, 2048),      # clusters of one to eight CTAs, chunk edges
    (2, 70000, 2048), (1, 300001, 1000), (160, 9000, 300),                # larger samples; more rows than SMs
])
@pytest.mark.parametrize("kind", ["normal", "clustered", "ties", "constant", "infinite"])
def test_topk_stage_over_row_lengths_and_distributions(rows, n, k, kind, sort):
    """Selection alone: the sampled bound, its failures (one value, values that are not finite, ties across the end of the
    selection) and the positions at which the row, the list and the chunks end. Ties go to the smaller position."""
    g = torch.Generator().manual_seed(n + k)
    stride = (n + 127) // 128 * 128
    sc = torch.randn(rows, stride, generator=g)
    if kind == "clustered":  # everything that is selected lies side by side
        sc[:, n // 3:n // 3 + 2 * k + 5] += 9.0
    elif kind == "ties":
        sc = (sc * 3).round() / 3 + 0.0
    elif kind == "constant":
        sc.fill_(0.25)
    elif kind == "infinite":
        sc[:, ::11] = float("-inf")
        sc[:, 5::997] = float("inf")
    sc[:, n:] = float("nan")  # never read as part of the row
    act = torch.full((rows,), n, dtype=torch.int32, device=DEV)
    out = torch.full((rows, 1, k), -7, dtype=torch.int32, device=DEV)
    pto.lightning_indexer_topk(sc.to(DEV), act, out, 1, k, sort=sort)
    torch.cuda.synchronize()
    assert pto.workspace_status()[0] == 0
    got = out.cpu()[:, 0].long()
    want = sc[:, :n].sort(dim=1, descending=True, stable=True).indices[:, :k]
    m = min(n, k)
    assert torch.all(got[:, m:] == -1)
    got = got[:, :m]
    if not sort:
        got, want = got.sort(dim=1).values, want.sort(dim=1).values
    assert torch.equal(got, want)


@pytest.mark.parametrize("sort", [True, False], ids=["ordered", "unordered"])
@pytest.mark.parametrize("n", [3001, 5120, 5121, 6148, 8193, 30001, 100003])  # rows that are lists, that are in one form only, longer ones
@pytest.mark.parametrize("kind", ["normal", "ties", "last"])
def test_many_rows_two_to_an_sm(kind, n, sort):
    """More rows than two per SM, in several rounds; every third row is short."""
    rows, k = 700, 2048
    g = torch.Generator(device=DEV).manual_seed(n)
    sc = torch.randn(rows, (n + 127) // 128 * 128, generator=g, device=DEV)
    if kind == "ties":
        sc = (sc * 3).round() / 3 + 0.0
    elif kind == "last":
        sc[:, n - 3000:n] += 20.0
    act = torch.full((rows,), n, dtype=torch.int32, device=DEV)
    act[::3] = torch.randint(1, n, (len(act[::3]),), generator=g, device=DEV, dtype=torch.int32)
    out = torch.full((rows, 1, k), -7, dtype=torch.int32, device=DEV)
    pto.lightning_indexer_topk(sc, act, out, 1, k, sort=sort)
    torch.cuda.synchronize()
    assert pto.workspace_status()[0] == 0
    inside = torch.arange(sc.shape[1], device=DEV)[None] < act[:, None]
    order = torch.where(inside, sc, -torch.inf).sort(dim=1, descending=True, stable=True).indices[:, :k]
    want = torch.where(torch.arange(k, device=DEV)[None] < act[:, None], order, -1)
    got = out[:, 0].long()
    if not sort:
        got, want = got.sort(dim=1).values, want.sort(dim=1).values
    assert torch.equal(got, want)


@pytest.mark.parametrize("sort", [True, False], ids=["ordered", "unordered"])
@pytest.mark.parametrize("rows,n", [(8, 32768), (40, 65536), (160, 20000), (3, 131072),  # clusters of 4, 2, 1 and 8 CTAs
                                    (1, 5000000)])  # a sample of its own size
@pytest.mark.parametrize("where", ["last", "runs", "aligned", "scattered"])
def test_neighbouring_positions_need_no_radix_select(where, rows, n, sort):
    """A selection of neighbouring positions (recency makes that the normal case) goes the same way as a scattered one."""
    k = 2048
    g = torch.Generator().manual_seed(n)
    sc = torch.randn(rows, n, generator=g)
    starts, run = {"last": ([n - k], k), "runs": ([n // 5 + 1, n // 3 + 7, n // 2 + 3, n - 700], 512),
                   "aligned": ([0, 4096, 8192, 16384], 512), "scattered": ([], 0)}[where]
    for at in starts:
        sc[:, at:at + run] += 20.0
    act = torch.full((rows,), n, dtype=torch.int32, device=DEV)
    out = torch.zeros((rows, 1, k), dtype=torch.int32, device=DEV)
    pto.reset_workspace_status()
    pto.lightning_indexer_topk(sc.to(DEV), act, out, 1, k, sort=sort)
    status = pto.workspace_status()
    assert status[0] == 0 and status[_lib.PTO_STATUS_RADIX_ROWS] == 0
    got, want = out.cpu()[:, 0].long(), sc.sort(dim=1, descending=True, stable=True).indices[:, :k]
    if not sort:
        got, want = got.sort(dim=1).values, want.sort(dim=1).values
    assert torch.equal(got, want)


@pytest.mark.parametrize("n", [640000, 655361, 900000, 983040, 1048576, 1500000])
def test_many_long_rows_need_no_radix_select(n):
    """More rows than SMs, around and beyond the length up to which two of them share an SM."""
    rows, k = 150, 2048
    g = torch.Generator(device=DEV).manual_seed(n)
    sc = torch.randn(rows, (n + 127) // 128 * 128, generator=g, device=DEV)
    act = torch.full((rows,), n, dtype=torch.int32, device=DEV)
    out = torch.zeros((rows, 1, k), dtype=torch.int32, device=DEV)
    pto.reset_workspace_status()
    pto.lightning_indexer_topk(sc, act, out, 1, k)
    status = pto.workspace_status()
    assert status[0] == 0 and status[_lib.PTO_STATUS_RADIX_ROWS] == 0
    got = out[:, 0].long()
    assert torch.equal(sc.gather(1, got), sc[:, :n].topk(k, dim=1).values)
    assert torch.all(got.sort(dim=1).values.diff(dim=1) > 0) and int(got.max()) < n


@pytest.mark.parametrize("sort", [True, False], ids=["ordered", "unordered"])
@pytest.mark.parametrize("rows,n", [(3, 5000), (8, 32768), (40, 65536), (160, 20000), (2, 1200000)])
@pytest.mark.parametrize("kind", ["outlier", "far_outliers", "tail", "masked", "infinite", "offset", "small"])
def test_uneven_scores_need_no_radix_select(kind, rows, n, sort):
    """Values far from the others must not send the others to one bin."""
    k = 2048
    g = torch.Generator().manual_seed(n)
    sc = torch.randn(rows, n, generator=g)
    if kind == "outlier":
        sc[:, 5] = 300.0
    elif kind == "far_outliers":
        sc[:, 5], sc[:, 7], sc[:, 4000] = 3e38, -3e38, 1e9
    elif kind == "tail":
        sc = (2.5 * sc).exp()
    elif kind == "masked":
        sc[:, ::7] = -1e4
        sc[:, 1::7] = torch.finfo(torch.float32).min
    elif kind == "infinite":
        sc[:, ::7] = float("-inf")
        sc[:, 1::997] = float("inf")
    elif kind == "offset":
        sc = sc + 1000.0
    elif kind == "small":
        sc = sc * 1e-20 - 1e-20
    act = torch.full((rows,), n, dtype=torch.int32, device=DEV)
    out = torch.zeros((rows, 1, k), dtype=torch.int32, device=DEV)
    pto.reset_workspace_status()
    pto.lightning_indexer_topk(sc.to(DEV), act, out, 1, k, sort=sort)
    status = pto.workspace_status()
    assert status[0] == 0
    # (of 1.2 million values 1204 are +inf, more than a bin holds; beside 3e38, 127 powers of two away, a bin is a 16th of one and
    # holds a thousand of those at the end of the selection)
    if n < 1000000 or kind not in ("infinite", "far_outliers"):
        assert status[_lib.PTO_STATUS_RADIX_ROWS] == 0
    got, want = out.cpu()[:, 0].long(), sc.sort(dim=1, descending=True, stable=True).indices[:, :k]
    if not sort:
        got, want = got.sort(dim=1).values, want.sort(dim=1).values
    assert torch.equal(got, want)


@pytest.mark.parametrize("n", [1, 700, 1999, 2048])
def test_nan_comes_first_in_a_row_that_is_selected_whole(n):
    g = torch.Generator().manual_seed(n)
    sc = torch.randn(2, 2048, generator=g)
    sc[0, n // 2], sc[1, n - 1] = float("nan"), float("inf")
    out = torch.zeros((2, 1, 2048), dtype=torch.int32, device=DEV)
    pto.lightning_indexer_topk(sc.to(DEV), torch.full((2,), n, dtype=torch.int32, device=DEV), out, 1, 2048)
    want = sc[:, :n].sort(dim=1, descending=True, stable=True).indices
    assert torch.equal(out.cpu()[:, 0, :n].long(), want) and torch.all(out[:, 0, n:] == -1)
