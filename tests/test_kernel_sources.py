"""CPU: what the kernel sources promise and no run can show reliably."""

import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _code(name):
    text = open(os.path.join(ROOT, "zmlx_b200", "csrc", name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def test_tensor_memory_matmul_reads_its_inputs_with_plain_loads():
    """Its kernels start while the kernels that write the plan, the token rows and the prepared rows still run.  Such data
    is not read-only for their lifetime, which the read-only load path (__ldg, or restrict-qualified inputs) requires;
    the weights, which are, come by TMA and cp.async."""
    code = _code("qmm_tma.cu")
    assert "pdl_wait" in code
    assert not re.search(r"__ldg|ld\.global\.nc|__restrict__", code)
