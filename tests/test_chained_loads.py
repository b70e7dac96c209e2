"""A kernel that may be resident while its inputs are still written (programmatic dependent launch) reads them through coherent
loads: ``__ldg``, ``ld.global.nc`` and ``const __restrict__`` parameters are for memory that nothing writes meanwhile, and the
compiler may move such loads above the wait.  The one file left out, skv_tc_prep.cu, reads only the inputs of a call whose first
kernel is launched plainly."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sparsespline_ffn_b200", "csrc")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name", sorted(os.path.basename(p) for p in glob.glob(os.path.join(CSRC, "*.cu*"))
                                        if not os.path.basename(p).startswith("skv_tc_prep")))
def test_no_read_only_loads_behind_a_wait(name):
    code = _code(name)
    assert "__ldg" not in code and "ld.global.nc" not in code
    for kernel in re.split(r"\b__global__\b", code)[1:]:
        if "pdl_wait()" in kernel:
            assert "__restrict__" not in kernel, kernel[:120]


def test_the_scan_is_launched_plainly():
    """What skv_tc_prep.cu reads through __ldg is complete before the first kernel of its chain starts."""
    assert re.search(r"tc_scan_kernel\s*<<<", _code("skv_tc_prep.cu"))
