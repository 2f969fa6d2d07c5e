"""The plain form of the step between sublayers against the general kernel (which an added zero vector selects), bit for bit."""
import pytest
import torch

from nanoflow_b200.ops import layer_list as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("kind", ["rms", "layer"])
@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("rows,cols,pad", [(1, 1024, 0), (5, 2048, 8), (149, 4096, 0), (2500, 4096, 4), (33, 8192, 64)])
def test_same_as_the_general_kernel(rows, cols, pad, bias, kind, dtype):
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    y, x = rand(rows, cols + pad).to(dtype), rand(rows, cols + pad)
    w = [rand(cols) for _ in range(4)]
    y[0, :cols] = 0.0
    if rows > 2:
        y[2, 3] = float("inf")
    norm = lambda i: (kind, w[i], w[i + 1] if bias else None)
    got = []
    for add in (None, torch.zeros(cols, device="cuda")):
        xx, h = x.clone(), torch.full((rows, cols + pad), 7.0, device="cuda", dtype=dtype)
        L.residual_norm(xx, y=y, norm_in=norm(0), add=add, h=h, norm_out=norm(2), cols=cols, eps=1e-5)
        got.append((xx, h))
    for a, b in zip(*got):
        assert torch.equal(a.nan_to_num(3.0, 4.0, 5.0), b.nan_to_num(3.0, 4.0, 5.0))
    assert torch.equal(got[0][0][:, cols:], x[:, cols:]) and (got[0][1][:, cols:] == 7).all()
