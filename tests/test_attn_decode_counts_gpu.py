"""Chunks of a context counted in words of the caller, and merged by the one that finishes last: the bits of the merge as a launch
of its own, again and again, whatever other callers run at the same time."""
import pytest
import torch

from nanoflow_b200 import ops
from nanoflow_b200.ops import layer_list as K

pytestmark = pytest.mark.gpu


# more chunks than a warp holds weights of at once (32); heads that share a warp; 64 columns; more (request, head) pairs than are
# counted (8192: two launches); requests of one chunk and of none beside the others
@pytest.mark.parametrize("B,kvh,group,hd,chunk_pages,max_chunks", [(3, 2, 4, 128, 1, 70), (24, 8, 8, 128, 3, 20), (7, 2, 16, 64, 2, 33),
                                                                   (300, 28, 1, 64, 2, 4), (400, 1, 2, 128, 5, 3)])
def test_same_bits_as_a_launch_of_its_own(B, kvh, group, hd, chunk_pages, max_chunks):
    g = torch.Generator(device="cuda").manual_seed(B)
    lens = [[0, 5, 40, 200, 1100][i % 5] + i % 37 for i in range(B)]
    counts, qh = [-(-n // 16) for n in lens], kvh * group
    P = sum(counts) + 2
    pool = torch.randn(P, 2, kvh, 16, hd, device="cuda", generator=g).bfloat16()
    kvi = torch.randperm(P, device="cuda", generator=g)[:sum(counts)].int()
    kvp = torch.tensor([0] + counts, device="cuda").cumsum(0).int()
    qo, st = torch.arange(B + 1, device="cuda").int(), ops.new_status()
    last = torch.tensor([(n - 1) % 16 + 1 if n else 0 for n in lens], device="cuda").int()
    q = torch.randn(B, qh * hd, device="cuda", generator=g).bfloat16()
    kw = dict(q_heads=qh, req_begin=0, req_count=B, status=st, chunk_pages=chunk_pages, max_chunks=max_chunks)
    ws = lambda: torch.full((B * qh * max_chunks * (hd + 2),), float("nan"), device="cuda")
    want = torch.zeros_like(q)
    ops.attn_decode(q, want, pool, qo, kvp, kvi, last, workspace=ws(), num_ctas=100, **kw)      # walked, merged by a second launch
    live = torch.tensor(lens, device="cuda") > 0
    for counts in [None] + [ops.decode_counts()] * 70:                                           # None: listed, a second launch too
        out = torch.zeros_like(q)
        ops.attn_decode(q, out, pool, qo, kvp, kvi, last, workspace=ws(), counts=counts, **kw)
        assert torch.equal(out[live], want[live]) and torch.isfinite(out[live].float()).all()
        assert counts is None or not counts.any()
    ops.check_status(st, "decode")


@pytest.mark.parametrize("counted", [False, True])
def test_two_forms_at_the_same_time(counted):
    """Two callers on two streams, with a plain and an extended launch that both start their form's counting: what one counts is
    nothing to the other."""
    B, kvh, group, hd, chunk_pages, max_chunks = 40, 8, 4, 128, 2, 24
    qh, lens = kvh * group, [17 * (i % 9) + 60 * (i % 4) + 1 for i in range(B)]
    g = torch.Generator(device="cuda").manual_seed(7)
    counts = [-(-n // 16) for n in lens]
    pool = torch.randn(sum(counts), 2, kvh, 16, hd, device="cuda", generator=g).bfloat16()
    kvi = torch.randperm(sum(counts), device="cuda", generator=g).int()
    kvp = torch.tensor([0] + counts, device="cuda").cumsum(0).int()
    qo, last = torch.arange(B + 1, device="cuda").int(), torch.tensor([(n - 1) % 16 + 1 for n in lens], device="cuda").int()
    q = torch.randn(B, qh * hd, device="cuda", generator=g).bfloat16()

    def plain(out, ws, own):
        ops.attn_decode(q, out, pool, qo, kvp, kvi, last, q_heads=qh, req_begin=0, req_count=B, chunk_pages=chunk_pages, max_chunks=max_chunks,
                        workspace=ws, counts=own)

    def extended(out, ws, own):
        K.paged_attention(q, pool, out, qo, kvp, kvi, last, heads=qh, scale=hd ** -0.5, req_count=B, chunk_pages=chunk_pages,
                          max_chunks=max_chunks, workspace=ws, counts=own)

    rounds, runs = 150, []
    for call in (plain, extended):
        ws = torch.empty(B * qh * max_chunks * (hd + 2), device="cuda")
        want = torch.zeros_like(q)
        call(want, ws, None)
        runs.append((call, want, ws, ops.decode_counts() if counted else None, torch.zeros(rounds, *q.shape, device="cuda", dtype=q.dtype), torch.cuda.Stream()))
    torch.cuda.synchronize()
    for i in range(rounds):
        for call, _, ws, own, outs, stream in runs:
            with torch.cuda.stream(stream):
                call(outs[i], ws, own)
    torch.cuda.synchronize()
    for _, want, _, own, outs, _ in runs:
        assert torch.isfinite(want.float()).all() and (outs == want).all()
        assert own is None or not own.any()


def test_counts_have_to_hold_every_pair():
    for bad in (torch.zeros(ops.DECODE_COUNTS - 1, device="cuda").int(), torch.zeros(ops.DECODE_COUNTS, device="cuda")):
        with pytest.raises(RuntimeError, match="counts"):
            ops._decode_counts(bad)
