"""Which calls the mid-rows GEMM kernel takes, and with how many parts of K (148 SMs)."""
from ctypes import byref, c_void_p

import pytest

from nanoflow_b200 import ops


def _plan(M, N, K, **f):
    p, out = ops.GemmParams(), ops.GemmPlan()
    p.M, p.N, p.K, p.workspace, p.workspace_bytes = M, N, K, c_void_p(256), 160 << 20
    for k, v in f.items():
        setattr(p, k, v)
    assert ops.lib().nfk_gemm_describe(byref(p), byref(out)) == 0
    return {n: getattr(out, n) for n, _ in ops.GemmPlan._fields_}


# us, tile kernel against mid-rows kernel, of each side of the line: beside the rule
@pytest.mark.parametrize("M,N,K,swiglu,parts", [(160, 8192, 28672, 0, 2), (288, 8192, 28672, 0, 2), (384, 8192, 28672, 0, 2), (160, 8192, 8192, 0, 2),
                                                (333, 8192, 8192, 0, 2), (700, 8192, 28672, 0, 1), (288, 4096, 14336, 0, 3), (333, 4096, 4096, 0, 0),
                                                (256, 14336, 4096, 1, 0), (333, 14336, 4096, 1, 0), (1100, 8192, 28672, 0, 0), (2048, 4096, 4096, 0, 0)])
def test_the_mid_rows_kernel_gets_the_sizes_at_which_it_is_faster(M, N, K, swiglu, parts):
    assert _plan(M, N, K, epilogue=swiglu)["mid_rows"] == parts
    for pin in (dict(tile_n=128), dict(num_ctas=100), dict(smem_budget_kb=130), dict(rows_kernel=2), dict(groups=2)):
        assert not _plan(M, N, K, epilogue=swiglu, **pin)["mid_rows"]


@pytest.mark.parametrize("swiglu", [0, 1])
def test_the_mid_rows_kernel_cuts_k_as_the_kept_order_does(swiglu):
    seen = 0
    for N, K in ((4608, 4096), (4096, 4096), (4096, 14336), (14336, 4096), (8192, 8192)):
        for M in range(97, 1100, 13):
            pl = _plan(M, N, K, epilogue=swiglu, keep_order=1)
            assert pl["mid_rows"] in (0, pl["split_k"]) and not (pl["mid_rows"] and pl["stream_k"])
            seen += pl["mid_rows"] > 0
    assert seen
