"""x sigmoid(z) of the gated epilogues against the division that it stands for, in 32 bits: the header's own function, compiled
into a kernel that writes both."""
import ctypes
import subprocess

import pytest
import torch

from nanoflow_b200.ops.build import ARCH_FLAGS, KERNEL_DIR, NVCC, NVCC_FLAGS

pytestmark = pytest.mark.gpu

SOURCE = """
#include "gated_act.cuh"
__global__ void both(const float* x, const float* z, float* ours, float* divided, int n) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  ours[i] = nf::mul_sigmoid(x[i], z[i]);
  divided[i] = x[i] / (1.f + __expf(-z[i]));
}
extern "C" int run_both(const float* x, const float* z, float* ours, float* divided, int n) {
  both<<<(n + 255) / 256, 256>>>(x, z, ours, divided, n);
  return static_cast<int>(cudaDeviceSynchronize());
}
"""


@pytest.fixture(scope="module")
def run_both(tmp_path_factory):
    at = tmp_path_factory.mktemp("gated")
    (at / "both.cu").write_text(SOURCE)
    subprocess.run([NVCC, *ARCH_FLAGS, *NVCC_FLAGS, "-I", str(KERNEL_DIR), "-shared", str(at / "both.cu"), "-o", str(at / "both.so")], check=True)
    lib = ctypes.CDLL(str(at / "both.so"))

    def call(x, z):
        out = [torch.empty_like(x) for _ in range(2)]
        p = lambda t: ctypes.c_void_p(t.data_ptr())
        torch.cuda.synchronize()
        assert lib.run_both(p(x), p(z), p(out[0]), p(out[1]), ctypes.c_int(x.numel())) == 0
        return out
    return call


def _ordered(t):
    """Numbers of 32 bits as integers whose difference counts ulps."""
    i = t.contiguous().view(torch.int32).long()
    return torch.where(i < 0, -(i & 0x7fffffff), i)


@pytest.mark.parametrize("alpha", [1.0, 1.702])
def test_within_an_ulp_of_the_division(run_both, alpha):
    g = torch.Generator(device="cuda").manual_seed(3)
    size = 10.0 ** torch.empty(1 << 22, device="cuda").uniform_(-38, 38.5, generator=g)
    near = torch.empty(1 << 22, device="cuda").uniform_(-150, 150, generator=g)
    x = torch.cat([size, -size, near])
    ours, divided = run_both(x, alpha * x)
    assert ((_ordered(ours) - _ordered(divided)).abs() <= 1).all()
    # and as near to 64 bits as the division is: an ulp is at most 2^-23 of a value, and on average there is no difference
    live = torch.cat([size < 80, size < 80, near.abs() < 80])
    want = x.double() / (1 + torch.exp(-(alpha * x).double()))
    off = [((t.double() - want).abs() / want.abs().clamp(min=1e-37))[live] for t in (ours, divided)]
    assert off[0].max() <= off[1].max() * (1 + 1e-3) + 2.0 ** -23 and off[0].mean() <= off[1].mean() * (1 + 1e-3)


def test_ends_of_the_range(run_both):
    inf, big = float("inf"), torch.finfo(torch.float32).max
    x = torch.tensor([0.0, -0.0, inf, -inf, float("nan"), big, -big, 3.39e38, -3.39e38, 1e-45, -1e-45, 1e-40, 2.0 ** -126, 88.0, -88.0, -88.7,
                      -88.8, -104.0], device="cuda")
    ours, divided = run_both(x, x)
    assert torch.equal(ours.isnan(), divided.isnan())
    there = ~divided.isnan()
    assert ((_ordered(ours) - _ordered(divided)).abs() <= 1)[there].all()
