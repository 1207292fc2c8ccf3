"""What the compiler made of kernels whose times hang on it, from the report that the build keeps."""
import os
import re

import pytest

import slapo_b200

LOG = os.path.join(os.path.dirname(slapo_b200.__file__), "csrc", "build", "ptxas.log")
ENTRY = re.compile(r"Compiling entry function '(?P<name>\w+)'.*?"
                   r"(?P<spill>\d+) bytes spill stores.*?Used (?P<regs>\d+) registers", re.S)


def _report():
    """{mangled name: (registers, spilled bytes)} of the newest build of each kernel."""
    if not os.path.exists(LOG):
        pytest.skip("no report of a build in this tree")
    with open(LOG) as f:
        return {m["name"]: (int(m["regs"]), int(m["spill"])) for m in ENTRY.finditer(f.read())}


@pytest.mark.parametrize("columns,stages", [(64, 8), (128, 6), (256, 4)])
@pytest.mark.parametrize("b_mn", [0, 1])
def test_plain_single_cta_product(columns, stages, b_mn):
    """Short products (tiles of 64 columns) went from 6.4 to 7.3 us when this kernel, its parameters grown by
    those of another epilogue, was compiled to 64 registers instead of 80."""
    want = f"gemm_tc05_kernelILi{columns}ELi{stages}ELb0ELb{b_mn}ELi0E"
    found = [v for k, v in _report().items() if want in k and "gemm2" not in k]
    if not found:
        pytest.skip("not part of the builds in the report")
    registers, spilled = found[-1]
    assert registers >= 80 and spilled == 0
