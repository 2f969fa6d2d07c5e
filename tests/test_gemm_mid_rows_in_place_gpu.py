"""The mid-rows GEMM with its residual in place: what it adds is requested ahead, over rounds of the same tile, while other
threads store."""
import pytest
import torch

from nanoflow_b200 import ops

pytestmark = pytest.mark.gpu


# one round, and two: 512 tokens are more than the ring holds at once; one and two tiles of tokens; columns that end inside a CTA's
@pytest.mark.parametrize("M,N,depth", [(33, 264, 1000), (300, 776, 2048), (480, 136, 1096), (512, 776, 2048), (700, 1024, 2048), (1000, 520, 2056)])
@pytest.mark.parametrize("split", [1, 2, 4])
def test_in_place_is_as_beside(M, N, depth, split):
    gen = torch.Generator(device="cuda").manual_seed(M + N + depth)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    a, w, c, bias = rn(M, depth).bfloat16(), (rn(N, depth) * depth ** -0.5).bfloat16(), rn(M, N).bfloat16(), rn(N).bfloat16()
    ws, st = torch.empty(16 << 20, device="cuda"), ops.new_status()
    kw = dict(beta=0.5, bias=bias, workspace=ws, rows_kernel=4, split_k=split, status=st)
    beside = ops.gemm(a, w, residual=c, **kw)
    for _ in range(3):
        out = c.clone()
        assert torch.equal(ops.gemm(a, w, out=out, residual=out, **kw), beside)
    ops.check_status(st, "gemm")
    want = a.double() @ w.double().T + 0.5 * c.double() + bias.double()
    # a bf16 rounding (2^-8), and sums of `depth` products of about depth^-1/2 in 32 bits
    assert ((beside.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all()
