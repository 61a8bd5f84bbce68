"""Two rules of the kernels that launch while the one before them drains,
checked in their source: a kernel lets the next one launch only once its own
predecessors have finished, and reads no field through the read-only path
(__ldg), since an earlier kernel may still be writing it when this one starts."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lqcd-dwf-hmc_b200", "csrc")


def _code(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def test_no_field_goes_through_the_read_only_path():
    for name in ("dwf_common.cuh", "dwf_chain.cuh", "dwf_hop.cuh", "field_ops.cu"):
        text = _code(name)
        # link records, which are complete before any launch that reads them
        text = re.sub(r"template <> struct LinkLoad<\w+> \{.*?\n\};", "", text, flags=re.S)
        text = re.sub(r"r\.l\d = __ldg\(lp[^;]*;", "", text)
        assert "__ldg" not in text, (name, re.findall(r"[^\n]*__ldg[^\n]*", text))


def test_dependents_launch_after_the_wait():
    n = 0
    for name in ("dwf_hop.cuh", "field_ops.cu"):
        text = _code(name)
        n += text.count("pdl_launch_dependents();")
        assert re.sub(r"pdl_wait\(\);\s*pdl_launch_dependents\(\);", "", text).count("pdl_launch_dependents();") == 0, name
    assert n >= 10
