"""Words between pinned host memory and the device, copied by a kernel."""
from ctypes import byref, c_void_p

import pytest
import torch

from nanoflow_b200 import ops
from nanoflow_b200.runtime.graph import WordCopyParams

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,skip", [(1, 0, 0), (0, 3, 0), (5, 1, 1), (1023, 4097, 0), (70001, 300001, 0), (4096, 7, 3)])
@pytest.mark.parametrize("to_host", [False, True])
def test_both_ways(n, m, skip, to_host):
    """Counts that are no multiple of four, addresses that are no multiple of 16 bytes (``skip``), nothing before or behind."""
    where = (lambda t: t.pin_memory()), (lambda t: t.cuda())
    put_src, put_dst = (where[1], where[0]) if to_host else where
    src = [put_src(torch.randint(0, 1 << 30, (k + 8,), dtype=torch.int32)) for k in (n, m)]
    dst = [put_dst(torch.full((k + 8,), -1, dtype=torch.int32)) for k in (n, m)]
    at = lambda t: c_void_p(t.data_ptr() + 4 * skip)
    p = WordCopyParams(dst=at(dst[0]), src=at(src[0]), count=n, dst2=at(dst[1]), src2=at(src[1]), count2=m)
    assert ops.lib().nfk_word_copy_p(byref(p), c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    for s, d, k in zip(src, dst, (n, m)):
        want = torch.full((k + 8,), -1, dtype=torch.int32)
        want[skip:skip + k] = s.cpu()[skip:skip + k]
        assert torch.equal(d.cpu(), want)


def test_bad_arguments():
    call = lambda **f: ops.lib().nfk_word_copy_p(byref(WordCopyParams(**f)), c_void_p(0))
    assert call(count=-1) == 1 and call(count=4) == 1 and call(count2=1) == 1 and call() == 0
