"""The kernels of one call overlap: a grid is resident while the kernel in front of it still writes what it is going to read.
Such memory is not read-only for the grid's lifetime, so no kernel of a chain may read it through the read-only path,
whose loads are free to move ahead of griddepcontrol.wait.  Nothing in a test on a GPU shows such a move until it happens."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "triton_int8_b200", "csrc")


def _code(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def test_no_read_only_loads_in_kernels_of_a_chain():
    quant, gemm = _code("quant.cu"), _code("gemm.cu")
    kernel = gemm[:gemm.index("sum_slots_kernel")]   # what follows is launched on its own
    assert "gemm_i8_kernel(" in kernel and "chain_wait();" in kernel
    for code in (quant, kernel, _code("common.cuh")):
        assert not re.search(r"__ldg\b|__ldcg\b|ld\.global\.nc|ld\.global\.L1::no_allocate\.nc", code)
