"""Split-K whose parts meet in a cluster: the same bits as the two launches that it stands for, at the edges of its tiles and
of K, with every form of the epilogue."""
import pytest
import torch

from nanoflow_b200 import ops
from nanoflow_b200.ops import layer_list as K

pytestmark = pytest.mark.gpu


def _operands(M, N, depth):
    gen = torch.Generator(device="cuda").manual_seed(M + N + depth)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    return rn(M, depth).bfloat16(), (rn(N, depth) * depth ** -0.5).bfloat16(), rn(M, N).bfloat16(), rn(N).bfloat16()


# rows around one, two and three tiles; columns that end inside a tile; K with a last part that is shorter and a last block that
# is not full; slices of 16, 32 ... 128 columns, the last of them narrower or empty
@pytest.mark.parametrize("M,N,depth,tile_n,cta_group,split", [
    (1, 256, 1024, 128, 1, 2), (97, 264, 1000, 96, 1, 3), (128, 4096, 4096, 256, 1, 8), (129, 520, 2056, 256, 2, 4), (256, 4096, 4096, 256, 2, 4),
    (255, 1000, 4096, 160, 2, 3), (257, 2048, 1096, 192, 2, 2), (333, 4096, 1536, 256, 2, 2), (640, 776, 2048, 64, 2, 4), (200, 96, 640, 32, 2, 4),
    (120, 512, 5 * 64, 256, 1, 4)])
@pytest.mark.parametrize("early", [False, True])
def test_same_bits_as_two_launches(M, N, depth, tile_n, cta_group, split, early):
    a, w, c, bias = _operands(M, N, depth)
    ws = torch.empty(max(16 << 20, split * M * N), device="cuda")
    outs = []
    for kernel in (2, 3):                              # 3: without the cluster
        st, out, norm = ops.new_status(), c.clone(), torch.empty_like(c)
        ops.gemm(a, w, out=out, residual=out, beta=0.5, bias=bias, workspace=ws, tile_m=1, tile_n=tile_n, cta_group=cta_group,
                 split_k=split, stream_k=2, rows_kernel=kernel, norm_w=bias, norm_out=norm, status=st, weights_ready=early,
                 early_start=ops.EARLY_FIRST | ops.EARLY_FURTHER if early else 0)
        ops.check_status(st, "gemm")
        outs.append((out, norm))
    assert torch.equal(outs[0][0], outs[1][0])
    want = a.double() @ w.double().T + 0.5 * c.double() + bias.double()
    # a bf16 rounding (2^-8), and sums of `depth` products of about depth^-1/2 in 32 bits
    assert ((outs[0][0].double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all()
    rows = outs[0][0].double()
    normed = rows * torch.rsqrt(rows.square().mean(-1, keepdim=True) + 1e-5) * bias.double()
    for _, norm in outs:
        assert ((norm.double() - normed).abs() <= normed.abs() * 2.0 ** -8 + 1e-6).all()


def test_rows_apart():
    a, w, c, bias = _operands(150, 520, 2048)
    ws = torch.empty(16 << 20, device="cuda")
    wide = torch.randn(150, 4096, device="cuda").bfloat16()
    kw = dict(workspace=ws, tile_m=1, tile_n=128, cta_group=2, split_k=3, stream_k=2)
    src = torch.zeros(150, 4104, device="cuda", dtype=torch.bfloat16)
    src[:, 8:2056] = a
    outs = [ops.gemm(src[:, 8:2056], w, out=wide.clone()[:, 40:560], rows_kernel=k, **kw) for k in (2, 3)]
    assert torch.equal(*outs) and torch.equal(outs[0], ops.gemm(a, w, rows_kernel=2, **kw))


@pytest.mark.parametrize("cta_group,split", [(1, 4), (2, 2)])
def test_blocks_on_the_diagonal_and_32_bit_columns(cta_group, split):
    a, w, _, _ = _operands(200, 4 * 136, 4 * 512)
    kw = dict(workspace=torch.empty(16 << 20, device="cuda"), tile_m=1, tile_n=64, cta_group=cta_group, split_k=split, stream_k=2)
    blocks = [K.gemm(a, w[:, :512].contiguous(), groups=4, group_k=512, k=512, rows_kernel=r, **kw) for r in (2, 3)]
    assert torch.equal(*blocks)
    want = torch.cat([a[:, 512 * i:512 * i + 512].double() @ w[136 * i:136 * i + 136, :512].double().T for i in range(4)], 1)
    assert ((blocks[0].double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all()
    wide = [torch.zeros(200, 344, device="cuda") for _ in range(2)]
    outs = [K.gemm(a, w, out32=o, f32_col0=200, lin_act="tanh", rows_kernel=r, **kw) for o, r in zip(wide, (2, 3))]
    assert torch.equal(*outs) and torch.equal(*wide)
    want = torch.tanh(a.double() @ w.double().T)
    assert ((wide[0].double() - want[:, 200:]).abs() <= 1e-4).all()
    assert ((outs[0].double() - want[:, :200]).abs() <= want[:, :200].abs() * 2.0 ** -8 + 1e-4).all()
