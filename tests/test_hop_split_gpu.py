"""The hop kernels of small lattices, which put the four axes on four warps, and
the direct ones: every mode and its dagger, every storage precision, against the CPU
oracle, where its blocks are ragged (sites not a multiple of a warp's), where
a warp has idle lanes (Ls 6, 12), on extents of 2 (one site is both
neighbours) and with each boundary phase; and a solve, whose block sums come
from this kernel's own number of blocks."""
import numpy as np
import pytest

from b200dwf import synth

pytestmark = pytest.mark.gpu

MODES = ["D", "Ddag", "DdagD", "H", "Hdag", "Deo", "Doe"]
CASES = [
    ([4, 4, 4, 4], 4, 1.0, 0.0, (1, 1, 1, -1)),
    ([6, 2, 4, 10], 6, 1.5, 0.5, (1, -1, 1, -1)),
    ([2, 6, 2, 6], 8, 1.0, 0.0, (-1, 1, 1, -1)),
    ([6, 4, 2, 6], 12, 1.5, 0.5, (1, 1, -1, 1)),
    ([4, 2, 6, 4], 16, 1.0, 0.0, (1, 1, 1, -1)),
]
# FP64 rounding of a few thousand operations; FP32 likewise.  Half storage rounds
# the input and up to four fields after it by at most 2^-12 (2^-9) of a slice's
# largest component, about three times their root mean square, uniformly (1 /
# sqrt 3 of it): 4.2e-4 (3.4e-3) each, times sqrt 5 and 1.7 for M_ee^-1.
TOL = {0: 1e-13, 1: 5e-6, 2: 1.6e-3, 3: 1.3e-2}


# 10: the split kernel (every case has at most one block an SM, its range); 0,
# 4: the direct kernel,
# whose FP64 links a warp stages for all its sites (at Ls 4 more of them than
# the epilogue's tile takes, at Ls 4 and 6 fewer lanes per site than directions)
@pytest.mark.parametrize("variant", ["10", "0", "4"])
@pytest.mark.parametrize("ci", range(len(CASES)))
def test_split_and_direct_hops_against_oracle(ci, variant, monkeypatch):
    import b200dwf
    from oracle.oracle import OracleDWF
    monkeypatch.setenv("B200_HOP_VARIANT", variant)
    lat, ls, b, c, bc = CASES[ci]
    u = synth.gauge_field(lat, 60 + ci, "hot")
    w = synth.spinor_field(lat, ls, 70 + ci)
    ora = OracleDWF(lat, ls, 0.04, 1.8, b, c, bc=bc)
    ora.set_links(u)
    op = b200dwf.DomainWall(lat, ls, 0.04, 1.8, b, c, bc=bc)
    op.set_config(u)
    for prec in range(4):
        fw, fv = op.new_field(prec), op.new_field(prec)
        op.convert(fw, w)
        for mode in MODES:
            for dag in (False, True):
                (op.mult_dag if dag else op.mult)(fv, fw, mode)
                ref = ora.mult(mode, w, dag)
                err = np.linalg.norm(op.reverse(fv) - ref) / np.linalg.norm(ref)
                assert err < TOL[prec], (prec, mode, dag, err)
    fb, fx = op.new_field(0), op.new_field(0)
    op.convert(fb, w)
    n, diff, rc = op.cg(fx, fb, 1e-20, 2000)
    xr, nr, _, rcr = ora.cg(w, 1e-20, 2000)
    assert rc == 0 and rcr == 0 and diff < 1e-9 and abs(n - nr) <= 2, (n, nr, diff)
    n, _, rc = op.shiftcg([op.new_field(0), op.new_field(0)], [0.0, 0.5], fb, 1e-20, 2000)
    assert rc == 0 and abs(n - nr) <= 2
