"""Arg-max over rows that are cut over the CTAs of a cluster: exact, the first of equal values, rows without a value."""
from ctypes import c_int, c_longlong, c_void_p

import pytest
import torch

from nanoflow_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows", [1, 2, 36, 37, 38, 73, 74, 75, 148, 149, 700])
@pytest.mark.parametrize("cols", [1, 7, 8, 16383, 16384, 32000, 32768, 65535, 128256])
def test_first_largest(rows, cols, dtype):
    ld = (cols + 7) // 8 * 8 + 8
    g = torch.Generator(device="cuda").manual_seed(rows * cols)
    x = torch.randn(rows, ld, device="cuda", generator=g).mul(4).round().to(dtype)[:, :cols]      # many equal values
    x[0, :] = float("-inf")
    if rows > 1:
        x[1, :] = float("nan")
    if rows > 2:
        x[2, :] = -1.0
        x[2, cols - 1] = float("inf")
    idx, val = torch.empty(rows, dtype=torch.int32, device="cuda"), torch.empty(rows, device="cuda")
    if dtype == torch.bfloat16:
        ops.argmax(x, idx_out=idx, val_out=val)
    else:
        assert ops.lib().nfk_argmax_f32(c_void_p(idx.data_ptr()), c_void_p(val.data_ptr()), c_void_p(x.data_ptr()), c_int(rows), c_int(cols),
                                        c_longlong(ld), c_int(0), c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    want = torch.arange(cols, device="cuda").expand(rows, cols).masked_fill(x != x.amax(dim=1, keepdim=True), cols).amin(dim=1).int()
    want[0] = cols // 8 * 8 if cols % 8 else 0          # no value above minus infinity: the first of the ragged end, if there is one
    want[1:2] = 0
    assert torch.equal(idx, want)
    assert torch.equal(val[2:], x.amax(dim=1).float()[2:]) and val[0] == float("-inf")
