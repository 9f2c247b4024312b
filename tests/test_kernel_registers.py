"""Registers of the stage kernels, from the compiler's report of the build: a pass that
streams HBM needs several blocks per SM, and one more array in a kernel body can cost
one of them."""
import pytest

REGS_PER_SM, THREADS = 65536, 256


def _blocks(ozlib, name):
    from ozaie_gb300 import build
    found = [r for k, r in build.kernel_registers("oz_split.cu").items() if name in k]
    if not found:
        pytest.skip("no compiler report (a library built elsewhere)")
    return [REGS_PER_SM // (-(-r // 8) * 8 * THREADS) for r in found]


def test_one_launch_split_with_norms_keeps_two_blocks_per_sm(ozlib):
    assert min(_blocks(ozlib, "k_exp_splitILi7ELb0ELb1E")) >= 2


def test_stage_pairs_keep_three_blocks_per_sm(ozlib):
    """Exponents or statistics of two operands, and their splits of one window and of two."""
    blocks = _blocks(ozlib, "k_stage_pairI")
    assert len(blocks) == 3 and min(blocks) >= 3
