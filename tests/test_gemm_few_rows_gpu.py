"""The GEMM kernel for few rows (csrc/kernels/gemm_few_rows.cuh) against the same product in fp32.

Tolerance: inputs are bf16, sums are fp32 and the result is rounded to bf16 once, so an element is off by at most half a
bf16 step of its own size (2^-9) plus the fp32 rounding of its sum, K * 2^-24 of the sum of absolute products at worst."""
import pytest
import torch

from nanoflow_b200 import ops

pytestmark = pytest.mark.gpu
F32 = torch.float32


def _data(M, N, K, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    return a, w


def _exact(a, w):
    return a.double() @ w.double().T, a.double().abs() @ w.double().abs().T


def _close(out, ref, size, K):
    bound = ref.abs() * 2 ** -8 + size * (K * 2.0 ** -24) + 1e-30
    worst = ((out.double() - ref).abs() / bound).max().item()
    assert worst <= 1.0, worst


@pytest.mark.parametrize("cg", [1, 2])
@pytest.mark.parametrize("split", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("M", [1, 2, 15, 16, 17, 33, 100, 128, 129, 200, 256, 257, 333])
def test_linear_edges(M, split, cg):
    if split * cg > 8 or (cg == 1 and M > 256):
        pytest.skip("not a form that the launcher builds")
    for N, K in ((8, 64), (264, 520), (384, 2048), (1000, 1096)):
        a, w = _data(M, N, K)
        if split > (K + 63) // 64:
            continue
        out = ops.gemm(a, w, rows_kernel=1, split_k=split, cta_group=cg)
        _close(out, *_exact(a, w), K)


@pytest.mark.parametrize("M", [1, 24, 96, 128, 250])
def test_bias_residual_norm(M):
    N, K = 1536, 1024
    a, w = _data(M, N, K)
    bias, res, nw = torch.randn(N, device="cuda").bfloat16(), torch.randn(M, N, device="cuda").bfloat16(), torch.rand(N, device="cuda").bfloat16()
    out, normed = res.clone(), torch.empty_like(res)
    ops.gemm(a, w, out=out, residual=out, bias=bias, rows_kernel=1, norm_w=nw, norm_out=normed)
    ref, size = _exact(a, w)
    _close(out, ref + bias.double() + res.double(), size + res.double().abs() + bias.double().abs(), K)
    x = out.double()
    want = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * nw.double()
    assert ((normed.double() - want).abs() <= want.abs() * 2 ** -7 + 1e-6).all()


@pytest.mark.parametrize("M", [1, 16, 48, 127, 128, 160, 300])
@pytest.mark.parametrize("F,K", [(64, 128), (200, 520), (2048, 1024)])
def test_gated(M, F, K):
    a, wg = _data(M, F, K)
    _, wu = _data(M, F, K, 1)
    for cg in (1, 2):
        if cg == 1 and M > 256:
            continue
        out = ops.gemm_swiglu(a, wg, wu, rows_kernel=1, cta_group=cg)
        g, u = a.double() @ wg.double().T, a.double() @ wu.double().T
        ref = torch.nn.functional.silu(g) * u
        # silu and the product carry the sums' errors; __expf adds a few fp32 steps
        assert ((out.double() - ref).abs() <= ref.abs() * 2 ** -8 + (g.abs() + u.abs() + 1) * 2 ** -14).all()


def test_same_sum_every_time_and_rows_independent():
    """The order of the sum depends on neither the run nor the rows beside it, and strided rows are read and written."""
    a, w = _data(128, 4096, 4096)
    one = ops.gemm(a, w, rows_kernel=1)
    for _ in range(5):
        assert torch.equal(one, ops.gemm(a, w, rows_kernel=1))
    wide, outw = torch.zeros(40, 4096 + 64, device="cuda").bfloat16(), torch.zeros(40, 4096 + 8, device="cuda").bfloat16()
    wide[:, :4096] = a[:40]
    ops.gemm(wide[:, :4096], w, out=outw[:, :4096], rows_kernel=1)
    assert torch.equal(outw[:, :4096], ops.gemm(a[:40].contiguous(), w, rows_kernel=1)) and not outw[:, 4096:].any()


def test_rule_gives_small_batches_to_it_and_keeps_other_forms():
    """With a workspace a small batch goes to it; without one, or with a pinned shape, to the tile kernel (one sum in the
    order of k, here the same for every width of the tile)."""
    a, w = _data(64, 2048, 1024)
    ws = torch.empty(1 << 22, device="cuda")
    assert torch.equal(ops.gemm(a, w, workspace=ws), ops.gemm(a, w, rows_kernel=1))
    plain = ops.gemm(a, w, rows_kernel=2)
    assert torch.equal(plain, ops.gemm(a, w)) and torch.equal(plain, ops.gemm(a, w, workspace=ws, tile_m=1, tile_n=128, split_k=1))
