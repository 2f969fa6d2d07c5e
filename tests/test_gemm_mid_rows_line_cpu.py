"""The line between the tile kernel and the mid-rows GEMM kernel, at sizes that were measured on both of its sides (148 SMs)."""
import pytest

from nanoflow_b200 import ops


# parts of K; 0: the tile kernel, which is faster there by 4 % and more
@pytest.mark.parametrize("M,N,K,gated,parts", [
    (288, 8192, 28672, 0, 2), (576, 8192, 28672, 0, 1), (288, 8192, 8192, 0, 2), (576, 8192, 8192, 0, 1), (576, 4096, 14336, 0, 2), (288, 32000, 8192, 0, 1),
    (288, 18944, 3584, 1, 1),
    (256, 8192, 28672, 0, 0), (512, 8192, 28672, 0, 0), (960, 8192, 28672, 0, 0), (1000, 8192, 28672, 0, 0), (1000, 8192, 8192, 0, 0), (160, 10240, 8192, 0, 0),
    (416, 10240, 8192, 0, 0), (333, 32000, 8192, 0, 0), (480, 32000, 8192, 0, 0), (896, 32000, 8192, 0, 0), (448, 128256, 4096, 0, 0), (960, 5120, 13824, 0, 0), (320, 5120, 5120, 0, 0), (416, 4096, 14336, 0, 0), (288, 4096, 4096, 0, 0), (288, 14336, 4096, 1, 0), (192, 2048, 8192, 0, 0),
    (333, 28672, 8192, 1, 0), (416, 28672, 8192, 1, 0), (896, 28672, 8192, 1, 0), (448, 22016, 8192, 1, 0), (700, 22016, 8192, 1, 0), (896, 18944, 3584, 1, 0)])
def test_each_side(M, N, K, gated, parts):
    assert ops.gemm_plan(M, N, K, swiglu=bool(gated), workspace_bytes=160 << 20)["mid_rows"] == parts


@pytest.mark.parametrize("M", [1, 16, 32])
def test_few_rows_of_a_head_in_kept_order(M):
    assert ops.gemm_plan(M, 128256, 4096, keep_order=True, workspace_bytes=160 << 20)["mid_rows"] == 0


@pytest.mark.parametrize("M,N,K", [(300, 32000, 8192), (333, 32000, 8192), (333, 128256, 4096)])
def test_some_rows_of_a_head_in_kept_order(M, N, K):
    """Whose other shape is four M tiles of 128 columns, half as fast."""
    plan = ops.gemm_plan(M, N, K, keep_order=True, workspace_bytes=160 << 20)
    assert plan["tile_m"] == 4 and plan["mid_rows"] == 1


@pytest.mark.parametrize("M,N,K", [(8, 4096, 4096), (64, 4096, 4096), (64, 4096, 14336), (96, 8192, 8192)])
def test_few_rows_without_a_workspace(M, N, K):
    assert ops.gemm_plan(M, N, K)["mid_rows"] == 1


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("N,K", [(28672, 8192), (22016, 8192), (8192, 28672), (4096, 4096), (5120, 13824)])
def test_k_is_cut_only_where_all_tiles_run_at_once(N, K, gated):
    for M in range(97, 1025, 29):
        parts = ops.gemm_plan(M, N, K, swiglu=gated, workspace_bytes=160 << 20)["mid_rows"]
        tiles = -(-N // (128 if gated else 256)) * (1 if M <= 512 else 2)
        assert parts < 2 or tiles <= {2: 35, 3: 22, 4: 14}[parts]
