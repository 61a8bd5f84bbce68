"""Launch errors on the fake CUDA runtime: a failed launch is reported by the
call that made it, and by no later one."""
import pytest

from fake_cuda import run


@pytest.mark.parametrize("mode", ["Deo", "Dee_inv"])     # a hop, a site-local map
def test_failed_launch_is_reported_once(tmp_path, mode):
    run(tmp_path, """
    u, pu = array(nlink)
    op = b200dwf.DomainWall([4, 4, 4, 4], 8, 0.1, 1.8)
    op.set_config(u)
    n = 24 * 128 * 8
    (w, pw), (v, pv) = array(n), array(n)
    mult = lambda: lib.b200_dwf_mult(op.handle, 0, pv, pw, b"%s", 0, None)
    b200dwf.check(mult())
    fake.fake_fail_launch(1)
    assert mult() != 0
    f, pf = array(nlink)
    b200dwf.check(lib.b200_momentum_update(lat, 0.1, pf, pu, None))
    b200dwf.check(mult())
    """ % mode)
