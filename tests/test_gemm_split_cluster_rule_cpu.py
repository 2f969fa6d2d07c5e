"""Which split-K shapes run as one launch whose parts meet in a cluster."""
import pytest

from nanoflow_b200 import ops


def _parts(M, N, K, tile_n, cta_group, split, **f):
    return ops.gemm_plan(M, N, K, tile_m=1, tile_n=tile_n, cta_group=cta_group, split_k=split, stream_k=2, workspace_bytes=160 << 20, **f)["cluster_parts"]


@pytest.mark.parametrize("M,N,K,tile_n,cta_group,split", [(1, 256, 1024, 128, 1, 2), (129, 520, 2056, 256, 2, 4), (128, 1024, 4096, 256, 1, 8), (640, 128, 2048, 64, 2, 4),
                                                          (128, 520, 4096, 128, 1, 7)])
def test_all_tiles_at_once(M, N, K, tile_n, cta_group, split):
    assert _parts(M, N, K, tile_n, cta_group, split) == split
    for pin in (dict(num_ctas=100), dict(smem_budget_kb=130)):
        assert _parts(M, N, K, tile_n, cta_group, split, **pin) == 0


@pytest.mark.parametrize("M,N,K,tile_n,cta_group,split", [(128, 16384, 4096, 256, 1, 8), (256, 16384, 4096, 256, 2, 4),     # more clusters of eight than fit
                                                          (120, 512, 5 * 64, 256, 1, 4), (128, 512, 9 * 64, 256, 1, 8),      # a part of K would be empty
                                                          (256, 512, 4096, 256, 2, 5), (128, 512, 8192, 128, 1, 9)])         # more than eight CTAs
def test_others_stay_two_launches(M, N, K, tile_n, cta_group, split):
    assert _parts(M, N, K, tile_n, cta_group, split) == 0
