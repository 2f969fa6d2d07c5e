"""The GEMM for a middling number of rows (weights as the tensor core's M operand, up to 512 tokens to a tile, K cut over a
cluster) against 64 bits and against the tile kernel, whose sums have the same order: the same bits."""
import pytest
import torch

from nanoflow_b200 import ops
from nanoflow_b200.ops import layer_list as L

pytestmark = pytest.mark.gpu

WS = 64 << 20


def _operands(M, N, depth):
    gen = torch.Generator(device="cuda").manual_seed(M + N + depth)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    return rn(M, depth).bfloat16(), (rn(N, depth) * depth ** -0.5).bfloat16(), (rn(N, depth) * depth ** -0.5).bfloat16(), rn(M, N).bfloat16(), rn(N).bfloat16()


# rows at the edges of an instruction's 32 tokens, of one and two instructions, of one and two tiles; columns that end inside a
# CTA's and inside a pair's; K with a last block that is not full and a last part that is shorter
SHAPES = [(1, 256, 1024), (31, 264, 1000), (33, 8, 512), (129, 520, 2056), (160, 4096, 4096), (255, 136, 1096), (256, 384, 2048), (257, 1000, 1536),
          (289, 2048, 1024), (333, 4096, 4096), (512, 776, 2048), (513, 520, 1024), (700, 1024, 2048), (1030, 264, 704)]


@pytest.mark.parametrize("M,N,depth", SHAPES)
@pytest.mark.parametrize("split", [1, 2, 3, 4])
@pytest.mark.parametrize("early", [False, True])
def test_linear(M, N, depth, split, early):
    a, w, _, c, bias = _operands(M, N, depth)
    ws, st = torch.empty(WS // 4, device="cuda"), ops.new_status()
    kw = dict(residual=c, beta=0.5, bias=bias, workspace=ws, split_k=split, status=st)
    norm = torch.empty_like(c)
    got = ops.gemm(a, w, rows_kernel=4, norm_w=bias, norm_out=norm, weights_ready=early,
                   early_start=ops.EARLY_FIRST | ops.EARLY_FURTHER if early else 0, **kw)
    ops.check_status(st, "gemm")
    assert torch.equal(got, ops.gemm(a, w, rows_kernel=3, tile_m=1, tile_n=128, stream_k=2, **kw))
    want = a.double() @ w.double().T + 0.5 * c.double() + bias.double()
    # a bf16 rounding (2^-8), and sums of `depth` products of about depth^-1/2 in 32 bits
    assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all()
    rows = got.double()
    normed = rows * torch.rsqrt(rows.square().mean(-1, keepdim=True) + 1e-5) * bias.double()
    assert ((norm.double() - normed).abs() <= normed.abs() * 2.0 ** -8 + 1e-6).all()


@pytest.mark.parametrize("M,N,depth", SHAPES)
@pytest.mark.parametrize("split", [1, 3])
def test_gated(M, N, depth, split):
    a, w, up, _, _ = _operands(M, N, depth)
    st = ops.new_status()
    got = ops.gemm_swiglu(a, w, up, rows_kernel=4, split_k=split, status=st)
    ops.check_status(st, "gemm")
    if split == 1:
        assert torch.equal(got, ops.gemm_swiglu(a, w, up, rows_kernel=2, tile_m=1, tile_n=128, stream_k=2))
    g, u = a.double() @ w.double().T, a.double() @ up.double().T
    want = g * torch.sigmoid(g) * u
    assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all()


def test_rows_apart():
    a, w, _, _, _ = _operands(150, 520, 2048)
    src, wide = torch.zeros(150, 4104, device="cuda", dtype=torch.bfloat16), torch.zeros(150, 4096, device="cuda", dtype=torch.bfloat16)
    src[:, 8:2056] = a
    got = ops.gemm(src[:, 8:2056], w, out=wide[:, 40:560], rows_kernel=4, split_k=2)
    assert torch.equal(got, ops.gemm(a, w, rows_kernel=4, split_k=2)) and not wide[:, :40].any() and not wide[:, 560:].any()


@pytest.mark.parametrize("M,N,depth,gated", [(160, 8192, 8192, False), (288, 4096, 14336, False), (700, 8192, 8192, False), (288, 28672, 2048, True)])
def test_the_rule_takes_it_and_the_order_is_kept(M, N, depth, gated):
    """Sizes on the rule's side of the line: the launch that the rule gives; with the order kept, the bits of the tile kernel."""
    a, w, up, _, _ = _operands(M, N, depth)
    ws = torch.empty(WS // 4, device="cuda")
    plan = ops.gemm_plan(M, N, depth, swiglu=gated, workspace_bytes=WS)
    run = lambda **kw: ops.gemm_swiglu(a, w, up, workspace=ws, **kw) if gated else ops.gemm(a, w, workspace=ws, **kw)
    if plan["mid_rows"]:
        assert torch.equal(run(), run(rows_kernel=4, split_k=plan["mid_rows"]))
    assert torch.equal(run(keep_order=True), run(keep_order=True, rows_kernel=2))


@pytest.mark.parametrize("split", [1, 3])
def test_32_bit_columns_and_activations(split):
    a, w, up, _, bias = _operands(300, 520, 1024)
    ws = torch.empty(WS // 4, device="cuda")
    wide = [torch.zeros(300, 320, device="cuda") for _ in range(2)]
    kw = dict(workspace=ws, split_k=split)
    outs = [L.gemm(a, w, out32=o, f32_col0=200, lin_act="relu2", rows_kernel=r, **kw, **t)
            for o, r, t in zip(wide, (4, 3), ({}, dict(tile_m=1, tile_n=64, stream_k=2)))]
    assert torch.equal(*outs) and torch.equal(*wide)
    if split == 1:
        for act in ("relu", "gelu_tanh"):
            got = [L.gemm(a, w, up=up, bias=bias, up_bias=bias, act=act, rows_kernel=r, **t) for r, t in ((4, {}), (2, dict(tile_m=1, tile_n=64)))]
            assert torch.equal(*got)
