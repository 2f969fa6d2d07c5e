"""Decode attention's counts: words of each engine, which its own launches use one after the other."""
import pytest
import test_graph_cpu as host

from nanoflow_b200.ops import DECODE_COUNTS, decode_counts
from nanoflow_b200.utils import depcheck


@pytest.mark.parametrize("pipeline_type,tp,nano", [("NON_OVERLAP_LOCAL", 1, None), ("LOCAL", 1, [16, 32]), ("PLLM", 2, [16, 16, 16])])
def test_decode_launches_count_in_memory_of_their_own_engine(pipeline_type, tp, nano, monkeypatch):
    """Work and finished chunks are counted in the engine's own words (two engines on one GPU may run at the same time), which
    the engine's own launches use one after the other."""
    make = host.Buffers
    monkeypatch.setattr(host, "Buffers", lambda **kw: make(**kw, decode_counts=decode_counts("cpu")))
    graphs = [host._host_graph(pipeline_type, tp, nano) for _ in range(2)]
    used = [{op.params.counts for op in g.ops if op.kernel == "nfk_attn_decode"} for g, _, _ in graphs]
    for (g, acc, (bufs, *_)), mine in zip(graphs, used):
        assert mine == {bufs.decode_counts.data_ptr()} and bufs.decode_counts.numel() >= DECODE_COUNTS
        assert not depcheck.check(g, acc)
        # launches that were not ordered would be seen
        at = [i for i, op in enumerate(g.ops) if op.kernel == "nfk_attn_decode"]
        g.ops[at[1]].stream, g.ops[at[1]].deps = "elsewhere", []
        assert any(at[1] in pair for pair in depcheck.check(g, acc))
    assert not used[0] & used[1]
