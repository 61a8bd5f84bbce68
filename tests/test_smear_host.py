"""Host code of the smearing plan on the fake CUDA runtime: which links
set_config reads in place and which it copies first."""
import pytest

from fake_cuda import run


@pytest.mark.parametrize("name,offset,kind,device,copied", [
    ("device memory on a 16-byte boundary", 0, "DEVICE", 0, False),
    ("device memory on an 8-byte boundary", 1, "DEVICE", 0, True),
    ("memory of another device", 0, "DEVICE", 1, True),
    ("page-locked host memory", 0, "HOST", 0, True),
])
def test_set_config_copies_what_its_kernel_cannot_read(tmp_path, name, offset, kind, device, copied):
    run(tmp_path, """
    sm = b200dwf.StoutSmear([4, 4, 4, 4], 0.1, 2)
    u, p = array(nlink, %d)
    fake.fake_pointer(p, %s, %d)
    log()
    b200dwf.check(lib.b200_smear_set_config(sm.handle, p, 1, None))
    lines = log()
    copies = [l for l in lines if l.startswith("memcpy") and hex(p.value) in l]
    launches = [i for i, l in enumerate(lines) if l.startswith("launch")]
    assert len(copies) == %d, lines
    # the planar copy and two levels, after the links have been copied
    assert len(launches) == 3, lines
    if copies:
        assert lines.index(copies[0]) < launches[0], lines
    """ % (offset, kind, device, int(copied)))


def test_level_copy_is_made_on_the_plans_device(tmp_path):
    """A level's lexical copy, made on the first request, is on the device of
    the plan whichever device the calling thread has current."""
    run(tmp_path, """
    sm = b200dwf.StoutSmear([4, 4, 4, 4], 0.1, 2)
    u, p = array(nlink)
    b200dwf.check(lib.b200_smear_set_config(sm.handle, p, 0, None))
    fake.fake_device(1)
    log()
    assert lib.b200_smear_config(sm.handle, 0)
    lines = log()
    assert any(l.startswith("malloc") for l in lines) and any(l.startswith("launch") for l in lines), lines
    for l in lines:
        if "device" in l:
            assert l.endswith("device 0"), lines
    d = ctypes.c_int(-1)
    fake.cudaGetDevice(ctypes.byref(d))
    assert d.value == 1
    """)


def test_host_copy_of_a_level_keeps_no_device_memory(tmp_path):
    """get_config of a level leaves the device memory in use as it was, also
    where there is none left for a copy in between, and puts the planar level in
    the lexical order."""
    run(tmp_path, """
    sm = b200dwf.StoutSmear([4, 4, 4, 4], 0.1, 2)
    u, p = array(nlink)
    b200dwf.check(lib.b200_smear_set_config(sm.handle, p, 0, None))
    used = fake.fake_used()
    for level in range(3):
        sm.config(level)
    assert fake.fake_used() == used
    fake.fake_limit(used)
    fake.fake_count()
    for level in range(2):
        got = sm.config(level)
        # entry k of link (mu, site) is double2 (9 mu + k) vol + site of its level
        mu, site, k, c = np.ix_(range(4), range(256), range(9), range(2))
        want = 2 * ((9 * mu + k) * 256 + site) + c
        got = got.reshape(4, 256, 9, 2)
        assert np.array_equal(got - got[0, 0, 0, 0], want), level
    assert fake.fake_used() == used
    """)
