"""Which kernel a GEMM of some hundred rows gets on this GPU, and that the launch is that kernel's."""
import pytest
import torch

from nanoflow_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,depth,gated,parts", [(288, 8192, 8192, False, 2), (576, 8192, 8192, False, 1), (288, 32000, 8192, False, 1), (288, 18944, 3584, True, 1),
                                                   (333, 4096, 4096, False, 0), (896, 18944, 3584, True, 0), (480, 32000, 8192, False, 0)])
def test_the_kernel_on_each_side(M, N, depth, gated, parts):
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    rn = lambda *s: (torch.randn(*s, device="cuda", generator=gen) * depth ** -0.25).bfloat16()
    a, w, ws = rn(M, depth), rn(N, depth), torch.empty(40 << 20, device="cuda")
    plan = ops.gemm_plan(M, N, depth, swiglu=gated, workspace_bytes=ws.numel() * 4)
    assert plan["mid_rows"] == parts
    up = rn(N, depth) if gated else None
    run = lambda **kw: ops.gemm_swiglu(a, w, up, workspace=ws, **kw) if gated else ops.gemm(a, w, workspace=ws, **kw)
    assert torch.equal(run(), run(rows_kernel=4, split_k=parts) if parts else run(rows_kernel=2))
