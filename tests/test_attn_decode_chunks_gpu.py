"""Decode attention over chunks of contexts of very different length: the list of chunks that a launch walks."""
import pytest
import torch

from nanoflow_b200 import ops
from nanoflow_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[1], [16, 0, 17], [0, 0, 700, 1, 0], [3000] + [5] * 40, [33 * (i % 7) + 1 for i in range(511)],
                                  [40 + i % 3 for i in range(512)], [20 + i % 50 for i in range(520)]])
@pytest.mark.parametrize("chunk_pages,max_chunks", [(1, 3), (8, 16), (40, 5)])
def test_every_chunk_is_taken_once(lens, chunk_pages, max_chunks):
    """Requests around the list's capacity (512), empty ones, and ones with more pages than the chunks cover, against the
    whole-context form of the same kernel. Both hold scores, weights and sums in fp32 and round the result to bf16 once, with
    the weights as bf16 in the products: an element is off by one bf16 step of the values' size at most."""
    B, kvh, group, hd = len(lens), 2, 4, 128
    qh = kvh * group
    g = torch.Generator(device="cuda").manual_seed(B)
    counts = [-(-n // 16) for n in lens]
    P = sum(counts) + 2
    pool = torch.randn(P, 2, kvh, 16, hd, device="cuda", generator=g).bfloat16()
    kvi = torch.randperm(P, device="cuda", generator=g)[:max(1, sum(counts))].int()
    kvp = torch.tensor([0] + counts, device="cuda").cumsum(0).int()
    qo = torch.arange(B + 1, device="cuda").int()
    last = torch.tensor([(n - 1) % 16 + 1 if n else 0 for n in lens], device="cuda").int()
    q = torch.randn(B, qh * hd, device="cuda", generator=g).bfloat16()
    whole, out = torch.zeros_like(q), torch.zeros_like(q)
    ws = torch.full((B * qh * max_chunks * (hd + 2),), float("nan"), device="cuda")
    st = ops.new_status()
    args = dict(q_heads=qh, req_begin=0, req_count=B, status=st)
    ops.attn_decode(q, whole, pool, qo, kvp, kvi, last, **args)
    ops.attn_decode(q, out, pool, qo, kvp, kvi, last, chunk_pages=chunk_pages, workspace=ws, max_chunks=max_chunks, **args)
    # with a CTA budget the launch keeps to its pipeline buffers and walks every (request, head, chunk) instead of a list
    walked = torch.zeros_like(q)
    ops.attn_decode(q, walked, pool, qo, kvp, kvi, last, chunk_pages=chunk_pages, workspace=ws, max_chunks=max_chunks, num_ctas=48, **args)
    ops.check_status(st, "decode")
    live = torch.tensor(lens, device="cuda") > 0
    assert torch.isfinite(out[live].float()).all() and torch.equal(out[live], walked[live])
    # weights of at most 1 and values of up to 4.5 standard deviations: 2^-8 of both, rounding at the end included
    assert ((out - whole)[live].float().abs() <= 4.5 * 2 ** -7).all()
