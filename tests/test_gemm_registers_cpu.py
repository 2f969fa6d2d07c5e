"""Registers of GEMM kernels, where they decide what runs side by side on an SM."""
import re
import subprocess

import pytest

from nanoflow_b200.ops.build import ARCH_FLAGS, KERNEL_DIR, NVCC, NVCC_FLAGS

BANK = 16384                                   # an SM's registers are four banks, one to a scheduler
GEMM_WARPS = 2                                 # most of the six warps of a CTA that share a bank


@pytest.fixture(scope="module")
def log(tmp_path_factory):
    return subprocess.run([NVCC, *ARCH_FLAGS, *NVCC_FLAGS, "-Xptxas", "-v", "-I", str(KERNEL_DIR), "-c", str(KERNEL_DIR / "gemm.cu"),
                           "-o", str(tmp_path_factory.mktemp("registers") / "gemm.o")], capture_output=True, text=True, check=True).stderr


def test_a_linear_gemm_leaves_registers_for_its_neighbours(log):
    # gemm_tcgen05_kernel<M tiles, epilogue, CTAs per tile, wide> with epilogue 0 (mangled: Li1ELi0E...)
    found = re.findall(r"entry function '\S*gemm_tcgen05_kernelILi(\d)ELi0ELi(\d)ELb(\d)E\S*' for.*?(\d+) bytes spill stores.*?Used (\d+) registers", log, re.S)
    assert len(found) == 5                     # 1, 2 and 4 M tiles; pairs; pairs with wide tiles
    for m_tiles, ctas, wide, spilled, regs in found:
        left = BANK - GEMM_WARPS * 32 * (-(-int(regs) // 8) * 8)
        # two CTAs of four warps with 152 registers a thread (a collective without a norm), or with several M tiles 136
        need = 2 * 32 * (152 if m_tiles == "1" else 136)
        assert int(spilled) == 0 and left >= need, (m_tiles, ctas, wide, regs)


def test_a_gated_gemm_takes_no_more_than_120(log):
    found = re.findall(r"entry function '\S*gemm_tcgen05_kernelILi1ELi1ELi(\d)ELb0E\S*' for.*?(\d+) bytes spill stores.*?Used (\d+) registers", log, re.S)
    assert len(found) == 2 and all(int(spilled) == 0 and int(regs) <= 120 for _, spilled, regs in found)


def test_the_second_pass_of_split_k_keeps_four_blocks_on_an_sm(log):
    spilled, regs = re.search(r"entry function '\S*splitk_reduce_kernel\S*' for.*?(\d+) bytes spill stores.*?Used (\d+) registers", log, re.S).groups()
    assert int(spilled) == 0 and 4 * 256 * int(regs) <= 4 * BANK
