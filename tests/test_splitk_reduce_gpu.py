"""The second launch of split-K with the norm of its rows folded in, at the edges of its groups of columns."""
import pytest
import torch

from nanoflow_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [512, 2048, 2056, 4096, 8192, 8200, 16384])
@pytest.mark.parametrize("split", [2, 5])
def test_second_launch_with_norm(N, split):
    """Groups of columns per thread: 1, 2, 4, 8, the last of them partly empty; more pieces than are requested at once."""
    M, depth = 140, 1024
    gen = torch.Generator(device="cuda").manual_seed(N)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    a, w, c, bias = rn(M, depth).bfloat16(), (rn(N, depth) * depth ** -0.5).bfloat16(), rn(M, N).bfloat16(), rn(N).bfloat16()
    ws, norm = torch.empty(split * M * N, device="cuda"), torch.empty_like(c)
    out = ops.gemm(a, w, residual=c, bias=bias, workspace=ws, tile_m=2, tile_n=128, split_k=split, stream_k=2, norm_w=bias, norm_out=norm)
    want = a.double() @ w.double().T + c.double() + bias.double()
    # a bf16 rounding (2^-8), and sums of `depth` products of about depth^-1/2 in 32 bits
    assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all()
    rows = out.double()
    normed = rows * torch.rsqrt(rows.square().mean(-1, keepdim=True) + 1e-5) * bias.double()
    assert ((norm.double() - normed).abs() <= normed.abs() * 2.0 ** -8 + 1e-6).all()
