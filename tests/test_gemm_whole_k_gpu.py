"""Shapes that leave K whole add up in the order of k: the same bits from each of them, for any number of rows. The models
that keep their order of sums rely on it when they take a tuned shape."""
import pytest
import torch

from nanoflow_b200 import ops
from nanoflow_b200.ops import autotune

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("M", [96, 129, 700, 2000])
@pytest.mark.parametrize("N,K", [(1536, 4096), (2056, 1096)])
def test_every_whole_k_shape_gives_the_same_bits(M, N, K, swiglu):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w, up = ((torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16() for _ in range(2))
    ws = torch.empty(160 << 18, device="cuda")
    shapes = [c for c in autotune.candidates(M, N, K, swiglu) if c != autotune.AUTO and c["split_k"] == 1 and c["stream_k"] != 1]
    outs = [ops.gemm_swiglu(a, w, up, workspace=ws, **{k: v for k, v in c.items() if k != "split_k"}) if swiglu else
            ops.gemm(a, w, workspace=ws, **c) for c in shapes]
    assert len(outs) >= 3 and all(torch.equal(outs[0], o) for o in outs[1:])
