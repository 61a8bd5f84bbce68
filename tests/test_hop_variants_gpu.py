"""The hop variants that the autotuner chooses among in half storage differ in
how they fetch, not in what they compute: the packed kernels (two slices a
thread) give the same stored bytes, so do the one-slice kernels, and these two
groups and the split kernel of small lattices project, multiply and sum in FP32
and differ by the order of a few FP32 roundings only."""
import numpy as np
import pytest

from b200dwf import synth

pytestmark = pytest.mark.gpu

CASES = [([4, 6, 2, 6], 4), ([6, 2, 4, 10], 6), ([4, 4, 6, 6], 8), ([2, 6, 4, 6], 12), ([6, 4, 2, 6], 16)]
MODES = [("Deo", False), ("Deo", True), ("D", False), ("Ddag", False), ("DdagD", False), ("H", False)]
PACKED, SINGLE, SPLIT = ("5", "6", "8", "9"), ("0", "1", "2", "3", "4"), "10"
# Between the groups and the split kernel: sums that differ by ~2^-21 (a few dozen FP32 roundings)
# round to another stored neighbour, 2^-11 away (2^-8 in bfloat16), with
# probability 2^-10 (2^-13), a root mean square of 2^-16 (2^-14.5) of a slice's
# largest component, which is about three times their root mean square; four
# stores and a factor 2 for M_ee^-1 give 2^-12.4 (2^-10.9).
TOL = {2: 2.0 ** -12, 3: 2.0 ** -10.5}


@pytest.mark.parametrize("prec", [2, 3])
@pytest.mark.parametrize("ci", range(len(CASES)))
def test_variants_share_one_arithmetic(ci, prec, monkeypatch):
    import b200dwf
    lat, ls = CASES[ci]
    op = b200dwf.DomainWall(lat, ls, 0.04, 1.8, 1.5, 0.5, bc=(1, -1, 1, -1))
    op.set_config(synth.gauge_field(lat, 80 + ci, "hot"))
    w, v = op.new_field(prec), op.new_field(prec)
    op.convert(w, synth.spinor_field(lat, ls, 90 + ci))
    out = {}
    for var in PACKED + SINGLE + (SPLIT,):
        monkeypatch.setenv("B200_HOP_VARIANT", var)
        for mode, dag in MODES:
            (op.mult_dag if dag else op.mult)(v, w, mode)
            out[var, mode, dag] = v.buf.cpu().numpy().copy(), op.reverse(v)
    for mode, dag in MODES:
        for group in (PACKED, SINGLE):
            for var in group[1:]:
                assert np.array_equal(out[var, mode, dag][0], out[group[0], mode, dag][0]), (var, mode, dag)
        a = out["0", mode, dag][1]
        for var in ("5", SPLIT):
            err = np.linalg.norm(a - out[var, mode, dag][1]) / np.linalg.norm(a)
            assert err < TOL[prec], (var, mode, dag, err)
