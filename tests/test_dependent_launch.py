"""The slice-pair GEMM may start while the kernel that writes its exponents, norms and
slices still runs (a programmatic dependent launch)."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "ozaie_gb300", "csrc")


def _code(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def test_gemm_reads_what_its_predecessor_writes_by_coherent_loads():
    """Non-coherent loads (ld.global.nc, __ldg) are for data that nothing writes while the
    kernel runs; the dependent launch breaks that for everything the stage kernels write."""
    code = _code("oz_gemm.cuh")
    assert "grid_wait_predecessor" in code
    for word in ("__ldg", "ld.global.nc", "__restrict__"):
        assert word not in code, word


def test_gemm_reads_nothing_of_its_predecessor_before_the_wait():
    """Before the wait the kernel touches its arguments, shared memory and TMEM only."""
    code = _code("oz_gemm.cuh")
    body = code[code.index("oz_gemm_kernel(const"):]
    head = body[:body.index("grid_wait_predecessor();")]
    for word in ("tile_ref", "g.er", "g.ec", "g.na", "g.nb,", "g.a_tiles", "g.b_tiles", "g.c", "g.err", "g.split_acc",
                 "g.split_cnt", "g.probs", "bulk_g2s"):
        assert not re.search(re.escape(word) + r"(?![A-Za-z_])", head), word
