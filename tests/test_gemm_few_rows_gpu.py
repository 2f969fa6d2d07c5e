"""The GEMM kernel for few rows (csrc/kernels/gemm_few_rows.cuh) against the same product in fp32.

Tolerance: inputs are bf16, sums are fp32 and the result is rounded to bf16 once, so an element is off by at most half a
bf16 step (8 significant bits: up to 2^-8 of its size) plus the fp32 rounding of its sum, K * 2^-24 of the sum of absolute
products at worst."""
from ctypes import byref, c_void_p

import pytest
import torch

from nanoflow_b200 import ops
from nanoflow_b200.ops import layer_list as forms
from nanoflow_b200.runtime.graph import NormParams

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


@pytest.mark.parametrize("few,most", [(40, 128), (1, 17), (150, 256)])
def test_same_sum_every_time_whatever_the_other_rows(few, most):
    """The order of the sum depends on neither the run nor, within 1 ... 128 and within 129 ... 256 rows (one CTA per tile and
    pairs of CTAs cut K differently), the number of rows beside a row; strided rows are read and written."""
    a, w = _data(most, 4096, 4096)
    one = ops.gemm(a, w, rows_kernel=1)
    for _ in range(5):
        assert torch.equal(one, ops.gemm(a, w, rows_kernel=1))
    assert torch.equal(one[:few], ops.gemm(a[:few], w, rows_kernel=1))
    wide, outw = torch.zeros(few, 4096 + 64, device="cuda").bfloat16(), torch.zeros(few, 4096 + 8, device="cuda").bfloat16()
    wide[:, :4096] = a[:few]
    ops.gemm(wide[:, :4096], w, out=outw[:, :4096], rows_kernel=1)
    assert torch.equal(outw[:, :4096], one[:few]) and not outw[:, 4096:].any()


@pytest.mark.parametrize("cg", [1, 2])
@pytest.mark.parametrize("N,K", [(136, 64), (384, 192), (1000, 1096), (4096, 4096)])
@pytest.mark.parametrize("M", [1, 40, 130])
def test_weights_fetched_before_the_rows_are_there(M, N, K, cg):
    """A chain of early launches: a norm writes the rows, the product has fetched weights meanwhile (fewer k-blocks than stages,
    and more), and the next norm writes the rows again. The same bits as one launch after the other."""
    g = torch.Generator(device="cuda").manual_seed(M)
    _, w = _data(1, N, K)
    _, up = _data(1, N, K, 1)
    ones = torch.ones(K, device="cuda").bfloat16()
    xs = [torch.randn(M, K, device="cuda", generator=g).bfloat16() for _ in range(8)]
    want = []
    for x in xs:
        a = ops.rmsnorm(x, ones, 1e-5)
        want.append((ops.gemm(a, w, rows_kernel=1, cta_group=cg), ops.gemm_swiglu(a, w, up, rows_kernel=1, cta_group=cg)))
    a = torch.empty_like(xs[0])
    got = [(torch.empty(M, N, device="cuda").bfloat16(), torch.empty(M, N, device="cuda").bfloat16()) for _ in xs]
    stream, early = c_void_p(torch.cuda.current_stream().cuda_stream), dict(rows_kernel=1, cta_group=cg, weights_ready=True, early_start=3)
    for _ in range(3):
        for x, (lin, gated) in zip(xs, got):
            p = NormParams(out=c_void_p(a.data_ptr()), x=c_void_p(x.data_ptr()), w=c_void_p(ones.data_ptr()), resid=c_void_p(0), rows=M,
                           cols=K, eps=1e-5, early_start=1)
            assert ops.lib().nfk_norm_p(byref(p), stream) == 0
            ops.gemm(a, w, out=lin, **early)
            ops.gemm_swiglu(a, w, up, out=gated, **early)
    torch.cuda.synchronize()
    assert all(torch.equal(p, q) and torch.equal(r, t) for (p, r), (q, t) in zip(want, got))


@pytest.mark.parametrize("M", [1, 33, 200])
@pytest.mark.parametrize("groups,n,K", [(1, 1000, 1096), (3, 200, 136), (8, 128, 64), (32, 512, 128)])
def test_other_forms_of_the_epilogue(M, groups, n, K):
    """Block-diagonal products, columns that leave as fp32, activations of finished columns."""
    g = torch.Generator(device="cuda").manual_seed(groups)
    a = torch.randn(M, groups * K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(groups * n, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    ref = torch.einsum("mgk,gnk->mgn", a.double().view(M, groups, K), w.double().view(groups, n, K)).reshape(M, -1)
    size = torch.einsum("mgk,gnk->mgn", a.double().abs().view(M, groups, K), w.double().abs().view(groups, n, K)).reshape(M, -1)
    kw = dict(groups=groups, group_k=K, k=K, rows_kernel=1)
    _close(forms.gemm(a, w, **kw), ref, size, K)
    for col0 in (0, 8, groups * n // 2 // 8 * 8):
        f32 = torch.zeros(M, groups * n - col0 + 4, device="cuda")
        out = forms.gemm(a, w, out32=f32, f32_col0=col0, **kw)
        assert ((f32[:, :groups * n - col0].double() - ref[:, col0:]).abs() <= size[:, col0:] * (K * 2.0 ** -24)).all()
        assert not f32[:, groups * n - col0:].any()
        if col0:
            _close(out, ref[:, :col0], size[:, :col0], K)
    relu2 = torch.relu(ref) ** 2            # the square doubles the sum's relative error
    got = forms.gemm(a, w, lin_act="relu2", **kw).double()
    assert ((got - relu2).abs() <= relu2 * 2 ** -8 + 2.1 * ref.abs() * size * (K * 2.0 ** -24) + (size * (K * 2.0 ** -24)) ** 2).all()


def test_rule_gives_small_batches_to_it_and_keeps_other_forms():
    """With a workspace a small batch goes to it; without one, or with a pinned shape, to the tile kernel (one sum in the
    order of k, here the same for every width of the tile)."""
    a, w = _data(64, 2048, 1024)
    ws = torch.empty(1 << 22, device="cuda")
    assert torch.equal(ops.gemm(a, w, workspace=ws), ops.gemm(a, w, rows_kernel=1))
    plain = ops.gemm(a, w, rows_kernel=2)
    assert torch.equal(plain, ops.gemm(a, w)) and torch.equal(plain, ops.gemm(a, w, workspace=ws, tile_m=1, tile_n=128, split_k=1))
