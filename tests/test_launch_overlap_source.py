"""A rule of the kernels that launch while the one before them drains, checked
in their source: a kernel lets the next one launch only once its own
predecessors have finished."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lqcd-dwf-hmc_b200", "csrc")


def _code(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def test_dependents_launch_after_the_wait():
    n = 0
    for name in ("dwf_hop.cuh", "field_ops.cu"):
        text = _code(name)
        n += text.count("pdl_launch_dependents();")
        assert re.sub(r"pdl_wait\(\);\s*pdl_launch_dependents\(\);", "", text).count("pdl_launch_dependents();") == 0, name
    assert n >= 10
