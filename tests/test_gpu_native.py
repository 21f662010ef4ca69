"""The native host path of the operators and the Python path behind it."""
import pytest
import torch

import pypto_b200 as pto
from pypto_b200 import _lib, ops
from pypto_b200 import inputs as gen

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _indexer(d, idx_query, out):
    pto.lightning_indexer_decode(idx_query, d.idx_query_scale, d.idx_key_cache, d.idx_key_scale, d.idx_weight, d.act_seq_key,
                                 d.block_table, out)


def test_a_call_keeps_its_workspace_until_it_returns():
    """Another thread may replace the stream's workspace while a call runs without the interpreter lock. Here the call's own error
    handler takes the entry away (the call is refused for its query's alignment, nothing is launched): the memory stays."""
    assert ops._native is not None
    d = gen.make_inputs([700], s1=1, seed=1, with_attention=False).to(DEV)
    out = torch.zeros((d.t, 1, 2048), dtype=torch.int32, device=DEV)
    _indexer(d, d.idx_query, out)  # (the workspace exists from here on)
    odd = torch.cat([d.idx_query.new_zeros(1), d.idx_query.reshape(-1)])[1:].reshape(d.idx_query.shape)
    torch.cuda.synchronize()
    key = (torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream)
    before = torch.cuda.memory_allocated()
    during = []

    def check(rc):
        del ops._workspaces[key]
        during.append(torch.cuda.memory_allocated())
        _lib.check(rc)

    ops._native.setup(ops._Handle, ops._workspaces, check)
    try:
        with pytest.raises(_lib.PtoError, match="aligned"):
            _indexer(d, odd, out)
    finally:
        ops._native.setup(ops._Handle, ops._workspaces, _lib.check)
    assert during == [before]
    assert torch.cuda.memory_allocated() < before  # nothing holds it any longer


@pytest.mark.parametrize("op", ["indexer", "indexer_bf16", "attention", "attention_packed", "fused", "fused_bf16", "prolog", "prolog_bf16"])
def test_both_host_paths_make_the_same_call(op, monkeypatch):
    """Every operator through the native path and through the Python checks behind it: the same results, bit for bit (ordered
    selections, so that nothing depends on the order in which a set is left)."""
    class Watched:
        def __init__(self, native):
            self.native, self.taken = native, []

        def __getattr__(self, name):
            return lambda *args: self.taken.append(getattr(self.native, name)(*args)) or self.taken[-1]

    def inputs():
        lens, bf = [700, 3000], torch.bfloat16
        if op.startswith("prolog"):
            make = gen.make_prolog_inputs if op == "prolog" else gen.make_prolog_nonquant_inputs
            return make([130, 200, 300], s1=1, seed=9, device=DEV)
        d = gen.make_nonquant_inputs(lens, seed=9) if op.endswith("bf16") else gen.make_inputs(lens, seed=9, with_topk=True)
        d = d.to(DEV)
        d.idx = torch.full((d.t, 1, 2048), -7, dtype=torch.int32, device=DEV)
        d.out = torch.zeros((d.b, 1, 128, 512), dtype=bf, device=DEV)
        return d

    def call(d):
        tail = lambda: (d.block_table, d.act_seq_key, d.out, 128, 1, 576 ** -0.5, 2048, 128, d.max_blocks)  # noqa: E731
        if op == "indexer":
            _indexer(d, d.idx_query, d.idx)
        elif op == "indexer_bf16":
            pto.lightning_indexer_topk_nonquant(d.idx_query, d.idx_key_cache, d.idx_weight, d.act_seq_key, d.block_table, d.idx)
        elif op == "attention":
            pto.sparse_flash_attention_quant_d(d.query_nope, d.query_rope, d.key_nope_2d, d.key_rope_2d, d.k_nope_scales,
                                               d.topk_indices, *tail())
        elif op == "attention_packed":
            rows = gen.pack_kv_rows(d.key_nope_2d, d.key_rope_2d, d.k_nope_scales)
            pto.sparse_attention_antiquant_d(d.query_nope, d.query_rope, rows, d.topk_indices, *tail())
        elif op == "fused":
            pto.decode_indexer_attention_quant(d.idx_query, d.idx_query_scale, d.idx_key_cache, d.idx_key_scale, d.idx_weight,
                                               d.query_nope, d.query_rope, d.key_nope_2d, d.key_rope_2d, d.k_nope_scales,
                                               d.act_seq_key, d.block_table, d.idx, d.out, sort=True)
        else:
            pto.decode_indexer_attention(d.idx_query, d.idx_key_cache, d.idx_weight, d.query_nope, d.query_rope, d.key_nope_2d,
                                         d.key_rope_2d, d.act_seq_key, d.block_table, d.idx, d.out, sort=True)
        return d.idx, d.out

    def prolog(p):
        t, bf = p["token_x"].shape[0], torch.bfloat16
        zeros = lambda shape, dt=bf: torch.zeros(shape, dtype=dt, device=DEV)  # noqa: E731
        q_nope, q_rope = zeros((t, 128, 512)), zeros((t, 128, 64))
        if op == "prolog":
            q_i8, q_sc, w = zeros((t, 64, 128), torch.int8), zeros((t, 64, 1), torch.float16), zeros((t, 64), torch.float16)
            caches = [p[k] for k in ("kv_cache", "kr_cache", "kv_scale_cache")] + [p["idx_k_cache"], p["idx_k_scale_cache"]]
            pto.mla_indexer_prolog_quant_d(
                *[p[k] for k in ("token_x", "w_dq", "w_uqqr", "w_qb_scale", "w_uk", "w_dkvkr", "gamma_cq", "gamma_ckv", "cos", "sin",
                                 "cache_index")], *caches[:3],
                *[p[k] for k in ("w_idx_qb", "w_idx_qb_scale", "w_idx_k", "w_idx_proj", "ln_gamma", "ln_beta", "hadamard_q",
                                 "hadamard_k")], *caches[3:], q_nope, q_rope, *caches[:3], q_i8, q_sc, *caches[3:], w, 1e-5, 1e-5)
            return q_nope, q_rope, q_i8, q_sc, w, *caches
        caches = [p[k] for k in ("kv_cache", "kr_cache", "idx_k_cache")]
        iq, w = zeros((t, 64, 128)), zeros((t, 64))
        pto.mla_indexer_prolog(*[p[k] for k in ("token_x", "w_dq", "w_uqqr", "w_uk", "w_dkvkr", "gamma_cq", "gamma_ckv", "cos", "sin",
                                                "cache_index")], *caches[:2],
                               *[p[k] for k in ("w_idx_qb", "w_idx_k", "w_idx_proj", "ln_gamma", "ln_beta")], caches[2], q_nope,
                               q_rope, iq, w)
        return q_nope, q_rope, iq, w, *caches

    run = prolog if op.startswith("prolog") else call
    run(inputs())  # (the workspace exists from here on)
    native, made = Watched(ops._native), []
    for path in (None, native):
        monkeypatch.setattr(ops, "_native", path)
        made.append(run(inputs()))
    torch.cuda.synchronize()
    assert native.taken == [True]
    for a, b in zip(*made):
        assert torch.equal(a, b)
