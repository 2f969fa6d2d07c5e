"""Which shape a GEMM call takes when the caller pins one that was measured at another number of rows."""
from ctypes import byref, c_void_p

import pytest
import torch

from nanoflow_b200 import ops
from nanoflow_b200.ops import autotune


def _plan(M, N, K, **f):
    p, out = ops.GemmParams(), ops.GemmPlan()
    p.M, p.N, p.K, p.workspace, p.workspace_bytes = M, N, K, c_void_p(256), 160 << 20
    for k, v in f.items():
        setattr(p, k, v)
    assert ops.lib().nfk_gemm_describe(byref(p), byref(out)) == 0
    return {n: getattr(out, n) for n, _ in ops.GemmPlan._fields_}


@pytest.mark.parametrize("tuned,M,holds", [(0, 48, True), (2048, 2048, True), (2048, 1793, True), (2048, 1792, False), (2048, 48, False),
                                           (256, 256, True), (256, 1, False), (256, 128, False), (256, 129, True), (256, 257, False),
                                           (100, 129, False), (128, 100, True), (128, 90, False), (90, 90, True)])
def test_a_tuned_shape_holds_for_its_own_number_of_row_groups(tuned, M, holds):
    """Up to 256 rows, where a tile of 128 rows is much: for its own number of such tiles, and not where the few-rows kernel
    takes the call unless the shape was measured at this very number of rows."""
    pin = dict(tile_m=1, tile_n=192, cta_group=1, split_k=1, stream_k=2)
    got = _plan(M, 10240, 8192, tuned_rows=tuned, **pin)
    assert got == (_plan(M, 10240, 8192, **pin) if holds else _plan(M, 10240, 8192))
    assert got["few_rows"] == (not holds and M <= 96)


@pytest.mark.parametrize("M", [1, 24, 96])
@pytest.mark.parametrize("swiglu", [0, 1])
def test_a_small_batch_takes_the_few_rows_kernel_whatever_the_dense_batch(M, swiglu):
    pin = dict(tile_m=1, tile_n=256, cta_group=2, split_k=1, stream_k=1)
    for tuned in (256, 1024, 2048):
        assert _plan(M, 28672, 8192, epilogue=swiglu, tuned_rows=tuned, **pin)["few_rows"]


@pytest.mark.parametrize("swiglu", [0, 1])
@pytest.mark.parametrize("M", [1, 64, 128, 129, 255, 256, 257, 333, 512, 513, 700, 1024, 2048, 4096, 16384])
@pytest.mark.parametrize("N,K", [(8, 64), (640, 512), (4096, 4096), (14336, 4096), (8192, 28672), (128256, 4096)])
def test_the_model_chooses_what_is_built(M, N, K, swiglu):
    pl = _plan(M, N, K, epilogue=swiglu)
    assert pl["stages"] >= 2 and pl["tile_m"] * pl["tile_n"] <= 512 and pl["smem_bytes"] <= 227 * 1024
    assert not (pl["cta_group"] == 2 and (M <= 128 or pl["tile_m"] != 1)) and not (swiglu and pl["split_k"] != 1)


def _cut(plan):
    """Where K is cut: tiles of the tail and their ranges, or the number of equal parts."""
    if plan["stream_k"]:
        return tuple(plan[k] for k in ("tile_m", "tile_n", "cta_group", "tail_first_tile", "tail_range_kb"))
    return plan["split_k"]


@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("N,K", [(4608, 4096), (4096, 4096), (12288, 4096), (4096, 14336), (14336, 4096), (64, 128)])
def test_no_pick_moves_the_cut_of_k_where_the_order_is_kept(N, K, swiglu):
    """Whatever the tuner offers at the dense batch, and whatever shape it would pin, K is cut as it is without a pick."""
    T, ws = 2048, 160 << 20
    every = autotune.candidates(T, N, K, swiglu)
    offered = autotune.same_order(every, T, N, K, swiglu, ws)
    assert autotune.AUTO in offered
    for M in (1, 96, 128, 700, 1793, 1840, 2000, 2048, 4096):
        want = _cut(ops.gemm_plan(M, N, K, swiglu=swiglu, workspace_bytes=ws, keep_order=True))
        for c in every:
            if c["split_k"] > 1 and swiglu:
                continue
            got = ops.gemm_plan(M, N, K, swiglu=swiglu, workspace_bytes=ws, keep_order=True, tuned_rows=T, **c)
            assert _cut(got) == want, (M, c, got)
    own = _cut(ops.gemm_plan(T, N, K, swiglu=swiglu, workspace_bytes=ws, keep_order=True))
    for c in offered:
        assert c == autotune.AUTO or (own == 1 and _cut(ops.gemm_plan(T, N, K, swiglu=swiglu, workspace_bytes=ws, keep_order=True, **c)) == 1)


@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("swiglu", [False, True])
def test_the_tuner_times_what_the_pipeline_launches(monkeypatch, swiglu, early):
    """Engines state that their weights are there, and kernels in line start early: so do the timed ones."""
    calls = []

    class Event:
        def __init__(self, enable_timing=True): pass
        record = synchronize = lambda self: None
        elapsed_time = lambda self, other: 1.0

    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(autotune, "gemm_swiglu" if swiglu else "gemm", lambda *a, **kw: calls.append(kw))
    a, w, out = torch.zeros(300, 128), torch.zeros(256, 128), torch.zeros(300, 256)
    r = autotune.tune_gemm(a, [w], out, weights_up=[w] if swiglu else None, early=early)
    assert r["best"] == autotune.AUTO and calls
    assert all(kw["weights_ready"] == early and kw["early_start"] == (3 if early else 0) for kw in calls)


@pytest.mark.parametrize("N,K,swiglu,last,not_at", [
    (4096, 4096, 0, 96, ()), (1280, 8192, 0, 64, ()), (32000, 8192, 0, 96, ()), (128256, 4096, 0, 48, ()),
    (14336, 4096, 1, 255, ()), (18944, 3584, 1, 255, ()), (2048, 4096, 1, 255, ()), (1024, 4096, 1, 160, ()),
    (22016, 8192, 1, 144, (128,)), (28672, 8192, 1, 144, (128,))])
def test_the_few_rows_kernel_gets_the_sizes_at_which_it_is_faster(N, K, swiglu, last, not_at):
    """The lines that the measurements beside the rule give (148 SMs)."""
    for M in (1, 16, 48, 64, 80, 96, 112, 127, 128, 129, 144, 145, 160, 192, 255, 256, 257, 300):
        assert _plan(M, N, K, epilogue=swiglu)["few_rows"] == (M <= last and M not in not_at), M
