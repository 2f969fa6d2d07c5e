"""Split-K whose parts meet in a cluster, with the launch that it takes named: the same bits as the two launches at the most
parts, the most tiles of rows and the slices that stay empty; shapes that it does not take."""
import pytest
import torch

from nanoflow_b200 import ops

pytestmark = pytest.mark.gpu


# eight parts of one CTA and four of a pair; three groups of rows, in pairs and in single CTAs; slices of 16 columns, and seven
# parts of 128 columns of which three own none; a last part of one block
@pytest.mark.parametrize("M,N,depth,tile_n,cta_group,split", [
    (128, 1024, 4096, 256, 1, 8), (100, 1000, 2504, 256, 1, 8), (255, 1024, 4096, 256, 2, 4), (640, 128, 2048, 64, 2, 4), (300, 264, 1000, 96, 1, 3),
    (128, 520, 4096, 128, 1, 7), (513, 192, 9 * 64, 32, 2, 2), (128, 2048, 9 * 64, 256, 1, 5)])
@pytest.mark.parametrize("early", [False, True])
def test_same_bits_as_two_launches(M, N, depth, tile_n, cta_group, split, early):
    gen = torch.Generator(device="cuda").manual_seed(M + N + depth)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    a, w, c, bias = rn(M, depth).bfloat16(), (rn(N, depth) * depth ** -0.5).bfloat16(), rn(M, N).bfloat16(), rn(N).bfloat16()
    ws = torch.empty(split * M * N, device="cuda")
    shape = dict(tile_m=1, tile_n=tile_n, cta_group=cta_group, split_k=split, stream_k=2)
    plan = ops.gemm_plan(M, N, depth, workspace_bytes=ws.numel() * 4, **shape)
    assert plan["cluster_parts"] == split and not plan["few_rows"] and not plan["mid_rows"]
    outs = []
    for kernel in (2, 3):                              # 3: without the cluster
        st, out, norm = ops.new_status(), c.clone(), torch.empty_like(c)
        ops.gemm(a, w, out=out, residual=out, beta=0.5, bias=bias, workspace=ws, rows_kernel=kernel, norm_w=bias, norm_out=norm, status=st,
                 weights_ready=early, early_start=ops.EARLY_FIRST | ops.EARLY_FURTHER if early else 0, **shape)
        ops.check_status(st, "gemm")
        outs.append(out)
    assert torch.equal(*outs)
    want = a.double() @ w.double().T + 0.5 * c.double() + bias.double()
    # a bf16 rounding (2^-8), and sums of `depth` products of about depth^-1/2 in 32 bits
    assert ((outs[0].double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all()
