"""The link-field kernels at the edges of their warps and lattices: volumes
that are not a multiple of a warp's 32 links, extents of 1 and 2 (a site is
its own neighbour, or the same one both ways), and arrays that only 8-byte
accesses can read, against plain numpy."""
import ctypes

import numpy as np
import pytest

from b200dwf import synth

pytestmark = pytest.mark.gpu

LATS = [[6, 2, 5, 3], [2, 1, 2, 3], [1, 4, 2, 2], [10, 6, 2, 4]]


def _cx(u, lat):
    return synth._as_complex(u, lat)


def _at(m):
    a = 0.5 * (m - synth._dag(m))
    return a - np.trace(a, axis1=-2, axis2=-1)[..., None, None] / 3.0 * np.eye(3)


def _to(f, mu, n=1):
    return np.roll(f, -n, axis=3 - mu)


def _loop(u, path):
    """Product of links along path (signed directions 1..4) from every site."""
    out = np.broadcast_to(np.eye(3), u.shape[1:]).astype(complex)
    off = [0, 0, 0, 0]

    def at(f):
        for d in range(4):
            f = _to(f, d, off[d])
        return f

    for s in path:
        mu = abs(s) - 1
        if s > 0:
            out = out @ at(u[mu])
            off[mu] += 1
        else:
            off[mu] -= 1
            out = out @ synth._dag(at(u[mu]))
    return out


@pytest.mark.parametrize("lat", LATS)
@pytest.mark.parametrize("rect", [0.0, -0.331])
def test_gauge_force_is_the_sum_of_its_loops(lat, rect):
    import b200dwf
    beta, cp = 2.13, 3.648
    u = synth.gauge_field(lat, 7, "hot")
    got = _cx(b200dwf.GaugeRect(lat, beta, cp, rect).force(u), lat)
    c = _cx(u, lat)
    for mu in range(4):
        m, s = mu + 1, 0
        for nu in range(4):
            if nu == mu:
                continue
            for n in (nu + 1, -nu - 1):
                # loops through U_mu(x), starting with it
                s = s + cp * _loop(c, [m, n, -m, -n])
                s = s + rect * (_loop(c, [m, m, n, -m, -m, -n]) + _loop(c, [m, n, n, -m, -n, -n]) +
                                _loop(c, [m, n, -m, -m, -n, m]))
        want = (-beta / 3.0) * _at(s)
        # up to 24 loops of 6 unitary products: 6 * 24 roundings of O(1) terms
        assert np.max(np.abs(got[mu] - want)) < 150 * 2.3e-16 * beta * (abs(cp) + 3 * abs(rect))


@pytest.mark.parametrize("lat", LATS)
@pytest.mark.parametrize("nsmear", [0, 1, 3])
def test_stout_levels(lat, nsmear):
    """Every level, the lower ones asked for after a first and refreshed by a
    second set_config."""
    import b200dwf
    sm = b200dwf.StoutSmear(lat, 0.1, nsmear)
    for seed in (3, 4):
        u = synth.gauge_field(lat, seed, "near", eps=0.3)
        sm.set_config(u)
        for level in range(nsmear + 1):
            want = synth.stout_smear(u, lat, 0.1, level)
            # hundreds of roundings a level on O(1) entries
            assert np.max(np.abs(sm.config(level) - want)) < 1e-13, (seed, level)


@pytest.mark.parametrize("lat", LATS)
def test_stout_jacobian_is_the_derivative(lat):
    """d Re tr(sigma U_smeared) along U -> exp(h A) U by central differences."""
    import b200dwf
    u = synth.gauge_field(lat, 5, "near", eps=0.3)
    sigma = synth.algebra_field(lat, 6)
    a = _cx(synth.algebra_field(lat, 8), lat)
    sm = b200dwf.StoutSmear(lat, 0.1, 2)
    sm.set_config(u)
    f = _cx(sm.jacobian(sigma), lat)
    c = _cx(u, lat)
    got = np.trace(f @ a @ c, axis1=-2, axis2=-1).real.sum()

    def s(h):
        # exp(h A) to fifth order: h = 1e-3, |A| ~ 3
        e = np.eye(3) + h * a + h * h / 2 * a @ a + h ** 3 / 6 * a @ a @ a + h ** 4 / 24 * a @ a @ a @ a
        v = _cx(synth.stout_smear(synth._as_real(e @ c), lat, 0.1, 2), lat)
        return np.trace(_cx(sigma, lat) @ v, axis1=-2, axis2=-1).real.sum()

    h = 1e-3
    d1, d2 = (s(h) - s(-h)) / (2 * h), (s(2 * h) - s(-2 * h)) / (4 * h)
    d = (4 * d1 - d2) / 3                  # O(h^4)
    assert abs(got - d) < 1e-6 * np.sqrt(c.size) * 3


@pytest.mark.parametrize("lat", LATS[:2])
@pytest.mark.parametrize("off", [0, 1])
def test_links_axpby_alignment(lat, off):
    """off = 1: arrays on an 8-byte boundary that is not a 16-byte one."""
    import torch
    import b200dwf
    n = 72 * int(np.prod(lat))
    g = torch.Generator().manual_seed(1)
    x = torch.randn(n + 2, dtype=torch.float64, generator=g).cuda()[off:off + n]
    y = torch.randn(n + 2, dtype=torch.float64, generator=g).cuda()[off:off + n]
    L = (ctypes.c_int * 4)(*lat)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    want = 1.25 * x - 0.5 * y                       # exact scalings: one rounding
    b200dwf.check(b200dwf.lib().b200_links_axpby(L, 1.25, p(x), -0.5, p(y), None))
    assert torch.max(torch.abs(y - want)).item() < 4 * 2.3e-16 * 4
    b200dwf.check(b200dwf.lib().b200_links_axpby(L, 2.0, p(x), 0.0, p(y), None))
    assert torch.equal(y, 2.0 * x)
    b200dwf.check(b200dwf.lib().b200_momentum_update(L, 0.5, p(x), p(y), None))
    assert torch.equal(y, 2.5 * x)


@pytest.mark.parametrize("lat", LATS[:2])
@pytest.mark.parametrize("off", [0, 1])
def test_stout_set_config_alignment(lat, off):
    """Device links on an 8-byte boundary that is not a 16-byte one smear to the
    same levels as host links."""
    import torch
    import b200dwf
    u = synth.gauge_field(lat, 3, "near", eps=0.3)
    d = torch.empty(u.size + 1, dtype=torch.float64, device="cuda")[off:off + u.size]
    d.copy_(torch.from_numpy(u))
    a, b = b200dwf.StoutSmear(lat, 0.1, 2), b200dwf.StoutSmear(lat, 0.1, 2)
    a.set_config(u)
    b200dwf.check(b200dwf.lib().b200_smear_set_config(b.handle, ctypes.c_void_p(d.data_ptr()), 1, None))
    for level in range(3):
        assert np.array_equal(a.config(level), b.config(level)), level


def test_gauge_force_under_capture():
    """A captured call, which reads the links where they are, replays to the
    same force as a direct one."""
    import torch
    import b200dwf
    lat = [6, 4, 2, 6]
    u = torch.from_numpy(synth.gauge_field(lat, 9, "hot")).cuda()
    L = (ctypes.c_int * 4)(*lat)
    a, b = torch.zeros_like(u), torch.zeros_like(u)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    call = b200dwf.lib().b200_gauge_force_rect
    b200dwf.check(call(L, 2.13, 3.648, -0.331, p(a), p(u), None))
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        b200dwf.check(call(L, 2.13, 3.648, -0.331, p(b), p(u), st))
    g.replay()
    torch.cuda.synchronize()
    assert torch.max(torch.abs(a - b)).item() < 1e-13
