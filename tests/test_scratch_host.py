"""The scratch that the gauge force keeps between calls, on the fake CUDA
runtime: bounded, given back on request and when its users are gone, and never
the reason for another allocation to fail."""
import pytest

from fake_cuda import run

FORCE = """
u, pu = array(nlink)
f, pf = array(nlink)
def force(l4=lat):
    b200dwf.check(lib.b200_gauge_force_rect(l4, 2.13, 3.648, -0.331, pf, pu, None))
force()
assert fake.fake_pool_idle() == 8 * nlink
"""

GIVEN_BACK = {
    "request": "b200dwf.check(lib.b200_scratch_release())",
    "GaugeRect": """
g = b200dwf.GaugeRect([4, 4, 4, 4], 2.13)
h = b200dwf.GaugeRect([4, 4, 4, 4], 2.13)
force()
del g
assert fake.fake_pool_idle() > 0        # h may use it
del h""",
    "plan": "op = b200dwf.DomainWall([4, 4, 4, 4], 8, 0.1, 1.8); force(); del op",
    "smearing plan": "sm = b200dwf.StoutSmear([4, 4, 4, 4], 0.1, 2); force(); del sm",
}


@pytest.mark.parametrize("how", GIVEN_BACK)
def test_scratch_is_given_back(tmp_path, how):
    run(tmp_path, FORCE + GIVEN_BACK[how] + """
assert fake.fake_pool_idle() == 0
force()                 # and kept again by the next user
assert fake.fake_pool_idle() == 8 * nlink
""")


def test_scratch_is_bounded(tmp_path):
    # 64 x 32 x 32 x 64 sites of 576 bytes are 2.4 GB
    run(tmp_path, FORCE + """
force((ctypes.c_int * 4)(64, 32, 32, 64))
assert 0 < fake.fake_pool_idle() <= 2 << 30
""")


def test_kept_scratch_fails_no_allocation(tmp_path):
    run(tmp_path, FORCE + """
b200dwf.check(lib.b200_scratch_release())
before = fake.fake_used()
op = b200dwf.DomainWall([4, 4, 4, 4], 8, 0.1, 1.8)
op.set_config(u)
need = fake.fake_used() - before
del op
force()
assert fake.fake_pool_idle() > 0
fake.fake_limit(fake.fake_used() + need)        # room for the plan alone
op = b200dwf.DomainWall([4, 4, 4, 4], 8, 0.1, 1.8)
op.set_config(u)
force()                                         # no room for scratch: still runs
fake.fake_limit(0)
for k in range(3):                              # really out of memory: an error
    assert lib.b200_dwf_create(ctypes.byref(ctypes.c_void_p()), lat, 8, 0.1, 1.8, None, None, 1.0, lat) == -3
b200dwf.check(lib.b200_momentum_update(lat, 0.1, pf, pu, None))     # and not this call's
""")
