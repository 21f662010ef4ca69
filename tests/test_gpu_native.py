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
