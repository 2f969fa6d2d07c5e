"""Activations of the gated GEMM epilogues, with gate and up values that arrive exactly: a row of A picks one column of the
weights. Each kernel that applies them, at the edges of its tiles."""
import pytest
import torch

from nanoflow_b200 import ops
from nanoflow_b200.ops import layer_list as K

pytestmark = pytest.mark.gpu

# (rows, columns, kwargs): few rows; single and pair tiles whose last chunk is 16 columns or the matrix's end; several M tiles;
# the stream-K tail with its second pass
FORMS = [(5, 1000, dict(rows_kernel=1)), (130, 136, dict(rows_kernel=1)), (128, 520, dict(rows_kernel=2, tile_m=1, tile_n=96)),
         (300, 1016, dict(rows_kernel=2, tile_m=1, tile_n=256, cta_group=2, stream_k=2)), (333, 264, dict(rows_kernel=2, tile_m=4, tile_n=128)),
         (700, 1000, dict(rows_kernel=2, tile_m=1, tile_n=224, cta_group=2, stream_k=1))]


def _act(kind, g, u):
    if kind == "relu":
        return g.clamp(min=0) * u
    if kind == "gelu_tanh":
        return 0.5 * g * (1 + torch.tanh(0.7978845608028654 * (g + 0.044715 * g ** 3))) * u
    if kind == "capped":
        g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0)
        return g / (1 + torch.exp(-1.702 * g)) * (u + 1.0)
    return g / (1 + torch.exp(-g)) * u


def _operands(M, N, depth=512):
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.zeros(M, depth, device="cuda", dtype=torch.bfloat16)
    a[torch.arange(M), torch.randint(0, depth, (M,), device="cuda", generator=gen)] = 1.0
    scale = 10.0 ** torch.empty(N, depth, device="cuda").uniform_(-4, 2.2, generator=gen)      # gates up to 150 either way
    wg = (torch.randn(N, depth, device="cuda", generator=gen) * scale).bfloat16()
    wu = torch.randn(N, depth, device="cuda", generator=gen).bfloat16()
    return a, wg, wu


@pytest.mark.parametrize("M,N,form", FORMS)
def test_silu_of_exact_gates(M, N, form):
    a, wg, wu = _operands(M, N)
    ws = torch.empty(64 << 18, device="cuda")
    got = ops.gemm_swiglu(a, wg, wu, workspace=ws, **form).double()
    pick = a.argmax(1)
    want = _act("silu", wg[:, pick].T.double(), wu[:, pick].T.double())
    # a bf16 rounding (2^-8); the argument of the exponential is rounded once more (150 x 2^-24); an exponential past the largest
    # number counts as infinite (90 x 5 x e^-88.7)
    assert ((got - want).abs() <= want.abs() * (2.0 ** -8 + 2e-5) + 2e-36).all()


@pytest.mark.parametrize("kind", ["silu", "relu", "gelu_tanh", "capped"])
@pytest.mark.parametrize("M", [40, 200, 300])
def test_every_activation(M, kind):
    a, wg, wu = _operands(M, 392)
    wg = wg.clamp(-30, 30)
    limits = dict(limit=7.0, alpha=1.702, shift=1.0) if kind == "capped" else {}
    got = K.gemm(a, wg, up=wu, act=kind, **limits).double()
    pick = a.argmax(1)
    want = _act(kind, wg[:, pick].T.double(), wu[:, pick].T.double())
    # tanh in 32 bits ends at one: 1 + tanh is off by up to 2^-24, times gate and up (30 x 5)
    tiny = 1e-5 if kind == "gelu_tanh" else 1e-30
    assert ((got - want).abs() <= want.abs() * (2.0 ** -8 + 2e-5) + tiny).all()
