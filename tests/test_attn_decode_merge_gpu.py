"""Chunks of a context merged by the one that finishes last: the bits of the merge as a launch of its own, again and again."""
import pytest
import torch

from nanoflow_b200 import ops

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
    for _ in range(70):                                                                          # every slot of the counts, and again
        out = torch.zeros_like(q)
        ops.attn_decode(q, out, pool, qo, kvp, kvi, last, workspace=ws(), **kw)
        live = torch.tensor(lens, device="cuda") > 0
        assert torch.equal(out[live], want[live]) and torch.isfinite(out[live].float()).all()
    ops.check_status(st, "decode")
