"""The work that users of this framework have it do, as timed cases.

Each case is one call (or the two or three calls that always come together) of
a hybrid Monte Carlo run on the public entry points: the even/odd domain-wall
operator in each storage precision, the solvers, the fermion force, the stout
smearing with its Jacobian and the gauge part of a molecular-dynamics step.
Sizes are the lattices of the repository's own configurations, tests and
benchmark (4^3x8 to 32^3x64, Ls 4 to 16), and ragged ones between them.

`exact` restates every path in plain torch complex arithmetic in 64 bits on
whole-lattice arrays, independent of the library's kernels.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch
import torch.utils.checkpoint

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "lqcd-dwf-hmc_b200"))

PRECS = {"f64": 0, "f32": 1, "f16": 2, "bf16": 3}
BC = (1, 1, 1, -1)
BETA, C_PLAQ, C_RECT = 2.13, 3.648, -0.331     # Iwasaki gauge action
RHO, NSMEAR = 0.1, 2                           # stout smearing of the fermion links
EPS = 0.01                                     # molecular-dynamics step


# ------------------------------------------------------------------ the cases
def _case(kind, lat, **kw):
    return dict({"kind": kind, "nx": lat[0], "ny": lat[1], "nz": lat[2], "nt": lat[3]}, **kw)


def _op(kind, lat, ls, prec="f64", mode="DdagD", mq=0.01, b=1.0, c=0.0, M0=1.8, **kw):
    return _case(kind, lat, ls=ls, prec=prec, mode=mode, mq=mq, b=b, c=c, M0=M0, **kw)


def listed():
    big, mid = (24, 24, 24, 48), (16, 16, 16, 32)
    return [
        # the smallest lattice that is run: one operator application of a test
        # or a debugging run, where launches and the wait for them are the time
        dict(_op("mult", (4, 4, 4, 8), 8), name="ddagd_f64_4x4x4x8"),
        # the headline: D_eo and its dagger in FP64 on the production lattice
        dict(_op("mult", big, 16, mode="Deo"), name="dslash_f64_24x24x24x48"),
        # the full operator in FP64 with Moebius coefficients on a ragged
        # lattice, Ls 12: residuals and Hamiltonians of a mid-size run
        dict(_op("mult", (14, 10, 6, 18), 12, b=1.5, c=0.5, M0=1.0, mq=0.02),
             name="ddagd_f64_moebius_14x10x6x18"),
        # the operator of the mixed-precision inner solves, half storage
        dict(_op("mult", big, 16, prec="f16"), name="ddagd_f16_24x24x24x48"),
        # the same in bfloat16 storage on the largest lattice that is run
        dict(_op("mult", (32, 32, 32, 64), 12, prec="bf16", mq=0.005), name="ddagd_bf16_32x32x32x64"),
        # the same in FP32, the inner precision of the reference's solver
        dict(_op("mult", mid, 16, prec="f32", b=1.5, c=0.5, M0=1.4), name="ddagd_f32_moebius_16x16x16x32"),
        # an FP64 CG solve on the published 8^4 Moebius run: many short launches
        dict(_op("cg", (8, 8, 8, 8), 12, mq=0.02, b=1.5, c=0.5, M0=1.0, tol2=1e-28), name="cg_f64_8x8x8x8"),
        # the strange quark's multishift solve, all poles of a rational at once
        dict(_op("shiftcg", mid, 16, mq=0.04, nshift=16, tol2=1e-20), name="multishift_16x16x16x32"),
        # a light-quark mixed-precision solve, half-storage inner CG
        dict(_op("richardson", mid, 16, prec="f16", tol2=1e-20), name="richardson_f16_16x16x16x32"),
        # the fermion force of one solution field
        dict(_op("force", big, 16), name="force_24x24x24x48"),
        # stout levels of new links and the force carried back through them
        dict(_case("smear", big), name="smear_24x24x24x48"),
        # the gauge part of a molecular-dynamics step: force, momenta, links
        dict(_case("gauge", mid), name="gauge_md_16x16x16x32"),
    ]


def _even(rng, lo, hi):
    """An even extent, spread over the logarithm of its range."""
    return 2 * max(1, round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2))


def draw(rng):
    kind = rng.choice(["mult"] * 6 + ["cg", "shiftcg", "richardson", "force", "smear", "gauge"])
    solve = kind in ("cg", "shiftcg", "richardson")
    top = 12 if solve else 28
    while True:
        lat = [_even(rng, 4, top) for _ in range(3)] + [_even(rng, 4, 1.5 * top)]
        if (8 if kind == "mult" else 512) <= math.prod(lat) <= 24 ** 3 * 48:
            break
    if kind in ("smear", "gauge"):
        return _case(kind, lat)
    ls = rng.choice([4, 6, 8, 12, 16])
    b, c, m0 = rng.choice([(1.0, 0.0, 1.8), (1.5, 0.5, 1.4)])
    kw = {"b": b, "c": c, "M0": m0, "mq": round(rng.choice([0.01, 0.04, 0.1, 1.0]) * (10 if solve else 1), 3)}
    kw["mq"] = min(kw["mq"], 1.0)
    if kind == "mult":
        return _op("mult", lat, ls, prec=rng.choice(["f64", "f64", "f32", "f16", "bf16"]),
                   mode=rng.choice(["Deo", "D", "Ddag", "DdagD", "DdagD", "H"]), **kw)
    if kind == "shiftcg":
        return _op(kind, lat, ls, nshift=rng.randint(4, 16), tol2=1e-20, **kw)
    if kind == "cg":
        return _op(kind, lat, ls, prec="f64", tol2=1e-20, **kw)
    if kind == "richardson":
        return _op(kind, lat, ls, prec=rng.choice(["f32", "f16", "bf16"]), tol2=1e-20, **kw)
    return _op(kind, lat, ls, **kw)


# ------------------------------------------------------------------ inputs
def _lat(case):
    return [case["nx"], case["ny"], case["nz"], case["nt"]]


def _vol(case):
    return math.prod(_lat(case))


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _links(case, gen, eps=0.3):
    """Smooth-to-rough SU(3) links: the first two rows of 1 + i eps H, H a
    Gaussian Hermitian matrix, orthonormalised, the third row completing
    them.  Reals in the lexical Field_G(Nvol, 4) layout."""
    n = 4 * _vol(case)
    g = torch.view_as_complex(torch.randn(n, 3, 3, 2, dtype=torch.float64, device="cuda", generator=gen))
    m = 0.5j * eps * (g + g.mH)
    m.diagonal(dim1=1, dim2=2).add_(1.0)
    r1 = m[:, 0] / torch.linalg.vector_norm(m[:, 0], dim=1, keepdim=True)
    r2 = m[:, 1] - (r1.conj() * m[:, 1]).sum(1, keepdim=True) * r1
    r2 = r2 / torch.linalg.vector_norm(r2, dim=1, keepdim=True)
    r3 = torch.linalg.cross(r1, r2).conj()
    return torch.view_as_real(torch.stack([r1, r2, r3], 1)).reshape(-1).contiguous()


def _algebra(case, gen):
    """Anti-Hermitian traceless Gaussian matrices (momenta) in that layout."""
    n = 4 * _vol(case)
    g = torch.view_as_complex(torch.randn(n, 3, 3, 2, dtype=torch.float64, device="cuda", generator=gen))
    h = 0.5 * (g + g.mH)
    tr = h.diagonal(dim1=1, dim2=2).sum(1).real / 3.0
    h.diagonal(dim1=1, dim2=2).sub_(tr[:, None])
    return torch.view_as_real(1j * h).reshape(-1).contiguous()


def _spinor(case, gen):
    """Gaussian Field(24, Nvol/2, Ls), every real N(0, 1)."""
    return torch.randn(24 * (_vol(case) // 2) * case["ls"], dtype=torch.float64, device="cuda", generator=gen)


def _shifts(case):
    """Poles of a rational on [1e-4, 10]: log-spaced, smallest first."""
    return np.geomspace(1e-4, 10.0, case["nshift"])


def prepare(case, seed):
    import b200dwf
    from b200dwf import hmc
    gen = _gen(seed)
    kind = case["kind"]
    st = {"case": case}
    u = _links(case, gen)
    if kind == "smear":
        st["dir"] = hmc.DirectorSmear(_lat(case), RHO, NSMEAR)
        st["u"], st["force"] = u, _algebra(case, gen)
        st["smeared"], st["sigma"] = torch.empty_like(u), torch.empty_like(u)
        st["lat"] = (ctypes.c_int * 4)(*_lat(case))
        return st
    if kind == "gauge":
        st["md"] = hmc.GaugeMD(_lat(case), BETA, C_PLAQ, C_RECT)
        st["u"], st["ip"] = u, _algebra(case, gen)
        return st
    op = b200dwf.DomainWall(_lat(case), case["ls"], case["mq"], case["M0"], case["b"], case["c"], 1.0, BC)
    hmc.GaugeMD.set_links(op, u)
    st["op"] = op
    prec = PRECS[case["prec"]] if kind == "mult" else 0
    st["w"] = op.new_field(prec)
    op.convert_device(st["w"], _spinor(case, gen))
    if kind == "mult":
        st["v"] = [op.new_field(prec) for _ in range(2 if case["mode"] == "Deo" else 1)]
    elif kind == "shiftcg":
        st["x"] = [op.new_field() for _ in range(case["nshift"])]
        st["sigma"] = _shifts(case)
    elif kind == "force":
        st["force"] = torch.empty_like(u)
    else:
        st["x"] = op.new_field()
    return st


# ------------------------------------------------------------------ one pass
def _values(field):
    """A field's stored numbers as tensors (no copy): FP64/FP32 storage whole;
    half storage as its scaled components and the scale of each (site, s)."""
    op, prec = field.op, field.prec
    if prec == 0:
        return field.buf.view(torch.float64)
    if prec == 1:
        return field.buf.view(torch.float32)
    col = field.buf.view(op.nvol, -1)
    k = 48 * op.Ls
    return [col[:, :k].view(torch.float16 if prec == 2 else torch.bfloat16), col[:, k:k + 4 * op.Ls].view(torch.float32)]


def run(state):
    import b200dwf
    from b200dwf import hmc
    case = state["case"]
    kind = case["kind"]
    if kind == "smear":
        lib, p = b200dwf.lib(), hmc._p
        d = state["dir"]
        d.set_config(state["u"])
        # the smeared links go to the operator's side, the force of the smeared
        # links arrives in sigma and is carried back to the thin ones
        lat, level = state["lat"], ctypes.c_void_p(d.config_ptr())
        b200dwf.check(lib.b200_links_axpby(lat, 1.0, level, 0.0, p(state["smeared"]), None))
        b200dwf.check(lib.b200_links_axpby(lat, 1.0, p(state["force"]), 0.0, p(state["sigma"]), None))
        d.jacobian(state["sigma"])
        b200dwf.check(lib.b200_force_mult_generator(lat, p(state["sigma"]), p(state["u"]), None))
        return [state["smeared"], state["sigma"]]
    if kind == "gauge":
        md = state["md"]
        md.update_p(state["ip"], state["u"], EPS)
        md.update_u(state["ip"], state["u"], EPS)
        return [state["ip"], state["u"]]
    op, w = state["op"], state["w"]
    if kind == "mult":
        v = state["v"]
        if case["mode"] == "Deo":
            op.mult(v[0], w, "Deo")
            op.mult_dag(v[1], w, "Deo")
        else:
            op.mult(v[0], w, case["mode"])
        return [_values(f) for f in v]
    if kind == "cg":
        _, _, rc = op.cg(state["x"], w, case["tol2"], 100000)
        b200dwf.check(rc)
        return [_values(state["x"])]
    if kind == "shiftcg":
        _, _, rc = op.shiftcg(state["x"], state["sigma"], w, case["tol2"], 100000)
        b200dwf.check(rc)
        return [_values(x) for x in state["x"]]
    if kind == "richardson":
        prec = PRECS[case["prec"]]
        _, _, _, rc = op.richardson(state["x"], w, prec, case["tol2"], 200, hmc.INNER_TOL2[prec], 100000)
        b200dwf.check(rc)
        return [_values(state["x"])]
    b200dwf.check(b200dwf.lib().b200_dwf_force_udiv(op.handle, hmc._p(state["force"]), w.ptr, None))
    return [state["force"]]


# ------------------------------------------------------------------ what a pass cannot do without
def _iterations(case):
    """Rough count of DdagD applications of a solve to its tolerance."""
    n = 480.0 / (1.0 + 14.0 * case["mq"]) * (1.3 if case["tol2"] < 1e-24 else 1.0)
    return min(n, 60.0 + 0.5 * 24 * _vol(case) ** 0.5)


def work(case):
    v = _vol(case)
    links = 72 * v * 8
    kind = case["kind"]
    if kind == "smear":
        # links in, force in; smeared links and force out; per level 6 staples
        # (2 products each) forward and back, the exponential's algebra
        return {"bytes": 4 * links, "flops": NSMEAR * 4 * v * 198 * (12 + 12 + 36 + 30)}
    if kind == "gauge":
        # links and momenta in and out; per link 6 plaquette and 18 rectangle
        # staples sharing their inner products, the exponential's 8 products
        return {"bytes": 4 * links, "flops": 4 * v * 198 * (6 * 2 + 18 * 2 + 8)}
    ls, half = case["ls"], v // 2
    size = {"f64": 8, "f32": 4, "f16": 2 + 4 / 24, "bf16": 2 + 4 / 24}
    mat = 1488.0 * ls * half                   # one D_eo
    chains = 24 * 22.0 * ls * half
    if kind == "mult":
        s = size[case["prec"]]
        field = 24 * ls * half * s
        lk = 72 * v * int(s)
        if case["mode"] == "Deo":
            return {"bytes": 3 * field + lk, "flops": 2 * mat}
        n = 4 if case["mode"] == "DdagD" else 2
        return {"bytes": 2 * field + lk, "flops": n * mat + (n + 1) * chains}
    field = 24 * ls * half * 8.0
    if kind == "force":
        return {"bytes": field + 2 * links, "flops": 3 * mat + 4 * chains + 4 * v * ls * 2 * 2 * 36 * 2}
    it = _iterations(case)
    n = case["nshift"] if kind == "shiftcg" else 1
    return {"bytes": (1 + n) * field + links, "flops": it * (4 * mat + 6 * chains + 24 * ls * half * (8 + 4 * (n - 1)))}


def tolerance(case):
    kind = case["kind"]
    if kind == "mult":
        return {"rel": {"f64": 1e-14, "f32": 1e-6, "f16": 1.6e-3, "bf16": 1.2e-2}[case["prec"]]}
    if kind in ("cg", "shiftcg", "richardson"):
        return {"rel": 1e-7}
    return {"rel": 1e-12}


# ------------------------------------------------------------------ the same in 64 bits, plain torch
# Whole-lattice arrays: spinors [s][t][z][y][x][spin][color], links
# [mu][t][z][y][x][row][col]; the array axis of direction mu in a
# [t][z][y][x] block is 3 - mu.  Dirac basis: gamma_mu as its two off-diagonal
# 2x2 blocks below, gamma_4 = diag(1, 1, -1, -1), gamma_5 swaps spin pairs.
_GAMMA = [
    {(0, 3): -1j, (1, 2): -1j, (2, 1): 1j, (3, 0): 1j},
    {(0, 3): -1.0, (1, 2): 1.0, (2, 1): 1.0, (3, 0): -1.0},
    {(0, 2): -1j, (1, 3): 1j, (2, 0): 1j, (3, 1): -1j},
    {(0, 0): 1.0, (1, 1): 1.0, (2, 2): -1.0, (3, 3): -1.0},
]


def _gamma(psi, mu):
    out = torch.empty_like(psi)
    for (i, j), c in _GAMMA[mu].items():
        out[..., i, :] = c * psi[..., j, :]
    return out


def _g5(psi):
    return psi[..., [2, 3, 0, 1], :]


def _color(u, psi):
    """u [...][3][3] on psi [s][...][spin][3], entry by entry."""
    out = torch.zeros_like(psi)
    for i in range(3):
        for j in range(3):
            out[..., i] += u[None, ..., i, j, None] * psi[..., j]
    return out


class _Exact:
    """The even/odd domain-wall operator on whole-lattice arrays."""

    def __init__(self, case, u_lex):
        nx, ny, nz, nt = _lat(case)
        self.case, self.ls = case, case["ls"]
        self.shape = (nt, nz, ny, nx)
        u = torch.view_as_complex(u_lex.reshape(4, nt, nz, ny, nx, 3, 3, 2)).clone()
        for mu in range(4):
            u[mu].select(3 - mu, self.shape[3 - mu] - 1).mul_(BC[mu])
        self.u = u
        t, z, y = torch.meshgrid(*(torch.arange(n, device="cuda") for n in (nt, nz, ny)), indexing="ij")
        self.odd = ((t + z + y) & 1)[..., None]
        x = torch.arange(nx // 2, device="cuda")
        # x of the half-lattice index ix2 on parity p: 2 ix2 + ((p + y + z + t) & 1)
        self.x = [2 * x + ((p + self.odd) & 1) for p in (0, 1)]
        ls, b, c, m = self.ls, case["b"], case["c"], case["mq"]
        hop = torch.zeros(2, ls, ls, dtype=torch.float64, device="cuda")
        for s in range(ls):
            hop[0, s, (s - 1) % ls] = 0.5 * (1.0 if s > 0 else -m)
            hop[1, s, (s + 1) % ls] = 0.5 * (1.0 if s < ls - 1 else -m)
        one = torch.eye(ls, dtype=torch.float64, device="cuda")
        a = 4.0 - case["M0"]
        self.m5 = b * one + 2.0 * c * hop
        self.inv = torch.linalg.inv((b * a + 1.0) * one + 2.0 * (c * a - 1.0) * hop)

    def fifth(self, mats, psi):
        """mats[0] on the + chirality, mats[1] on the -, along s."""
        up, dn = psi[..., :2, :], psi[..., 2:, :]
        flat = lambda v: torch.view_as_real(v.contiguous()).reshape(self.ls, -1)  # noqa: E731
        p = mats[0] @ flat(up + dn)
        q = mats[1] @ flat(up - dn)
        back = lambda v: torch.view_as_complex(v.reshape(*up.shape, 2))  # noqa: E731
        p, q = 0.5 * back(p), 0.5 * back(q)
        return torch.cat([p + q, p - q], dim=-2)

    def mat(self, name, dag):
        m = getattr(self, name)
        return m.transpose(1, 2) if dag else m

    def full(self, w, parity):
        """Field(24, Nvol/2, Ls) reals to a whole-lattice array, zero on the
        other parity."""
        nt, nz, ny, nx = self.shape
        half = torch.view_as_complex(w.reshape(self.ls, nt, nz, ny, nx // 2, 4, 3, 2))
        out = torch.zeros(self.ls, nt, nz, ny, nx, 4, 3, dtype=torch.complex128, device="cuda")
        for q in (0, 1):        # rows of one x offset at a time
            rows = self.odd[..., 0] == q
            out[:, rows, (parity + q) & 1::2] = half[:, rows]
        return out

    def half(self, psi, parity):
        """The sites of one parity, in the half-lattice order."""
        nt, nz, ny, nx = self.shape
        out = torch.empty(self.ls, nt, nz, ny, nx // 2, 4, 3, dtype=torch.complex128, device="cuda")
        for q in (0, 1):
            rows = self.odd[..., 0] == q
            out[:, rows] = psi[:, rows, (parity + q) & 1::2]
        return out

    def hop(self, psi):
        out = torch.zeros_like(psi)
        for mu in range(4):
            ax = 4 - mu         # the array axis with s in front
            f = _color(self.u[mu], torch.roll(psi, -1, ax))
            out += f - _gamma(f, mu)
            b = torch.roll(_color(self.u[mu].mH, psi), 1, ax)
            out += b + _gamma(b, mu)
        return out

    def deo(self, psi, dag=False):
        if dag:
            return self.fifth(self.mat("m5", True), -0.5 * _g5(self.hop(_g5(psi))))
        return -0.5 * self.hop(self.fifth(self.m5, psi))

    def D(self, psi):
        return psi - self.fifth(self.inv, self.deo(self.fifth(self.inv, self.deo(psi))))

    def Ddag(self, psi):
        i = self.mat("inv", True)
        return psi - self.deo(self.fifth(i, self.deo(self.fifth(i, psi), True)), True)

    def mult(self, mode, psi):
        if mode == "D":
            return self.D(psi)
        if mode == "Ddag":
            return self.Ddag(psi)
        if mode == "H":
            return _g5(self.D(psi)).flip(0)
        return self.Ddag(self.D(psi))

    def solve(self, b, sigma=0.0, tol2=1e-27):
        """CG on DdagD + sigma."""
        x, r = torch.zeros_like(b), b.clone()
        p, rr = r.clone(), _norm2(b)
        stop = tol2 * rr
        while rr > stop:
            q = self.Ddag(self.D(p)) + sigma * p
            a = rr / torch.view_as_real(p).flatten().dot(torch.view_as_real(q).flatten()).item()
            x += a * p
            r -= a * q
            new = _norm2(r)
            p = r + (new / rr) * p
            rr = new
        return x

    def force(self, eta):
        """Both halves of the force of eta, lexical Field_G reals."""
        dag = self.mat("inv", True)
        ye = self.fifth(self.m5, eta)
        yo = self.fifth(self.m5, self.fifth(self.inv, -0.5 * self.hop(ye)))
        ae = self.fifth(dag, self.D(eta))
        ao = self.fifth(dag, self.deo(ae, True))
        y, a = ye + yo, ae + ao        # the two parities of one array
        out = []
        for mu in range(4):
            ax = 4 - mu
            ph = torch.ones(self.shape, dtype=torch.float64, device="cuda")
            ph.select(3 - mu, self.shape[3 - mu] - 1).mul_(BC[mu])
            f = 0.0
            for near, here, sign in ((y, a, -1.0), (a, y, 1.0)):
                n = torch.roll(near, -1, ax)
                n = n + sign * _gamma(n, mu)
                f = f + torch.stack([torch.stack([(n[..., i] * here[..., j].conj()).sum((0, -1)) for j in range(3)], -1)
                                     for i in range(3)], -2)
            out.append(0.5 * ph[..., None, None] * f)
        return torch.view_as_real(torch.stack(out)).reshape(-1)

    def stored(self, half, prec):
        """A half-lattice array in a field's storage: per site 16-byte chunks
        (k, s), component q = color + 3 spin; half storage scaled by the
        largest magnitude of each (site, s)."""
        v = torch.view_as_real(half.contiguous()).reshape(self.ls, -1, 24).transpose(0, 1)   # [site][s][24]
        per = {"f64": 2, "f32": 4}.get(prec, 8)
        chunks = lambda w: w.reshape(w.shape[0], self.ls, 24 // per, per).transpose(1, 2).reshape(w.shape[0], -1)  # noqa: E731
        if per < 8:
            return chunks(v).reshape(-1).contiguous()
        top = v.abs().amax(2)
        return [chunks(v / top[..., None]).contiguous(), top.contiguous()]


def _norm2(psi):
    return torch.view_as_real(psi).flatten().square().sum().item()


def _su3(u_lex, lat):
    return torch.view_as_complex(u_lex.reshape(4, lat[3], lat[2], lat[1], lat[0], 3, 3, 2))


def _mul(*ms):
    """Products of 3x3 matrix fields, entry by entry."""
    out = ms[0]
    for b in ms[1:]:
        out = sum(out[..., :, k, None] * b[..., None, k, :] for k in range(3))
    return out


def _to(f, mu, n=1):
    """The field at x + n mu."""
    return torch.roll(f, -n, 3 - mu)


def _traceless(m):
    """Traceless anti-Hermitian part."""
    a = 0.5 * (m - m.mH)
    tr = a.diagonal(dim1=-2, dim2=-1).sum(-1) / 3.0
    return a - tr[..., None, None] * torch.eye(3, dtype=m.dtype, device=m.device)


def _stout(u):
    """One stout step of all four directions."""
    out = []
    for mu in range(4):
        c = 0.0
        for nu in range(4):
            if nu == mu:
                continue
            c = c + _mul(u[nu], _to(u[mu], nu), _to(u[nu], mu).mH)
            c = c + _to(_mul(u[nu].mH, u[mu], _to(u[nu], mu)), nu, -1)
        q = _traceless(_mul(RHO * c, u[mu].mH))
        # exp by its Taylor series on a quarter of the exponent, squared twice
        e = term = torch.eye(3, dtype=q.dtype, device=q.device).expand(q.shape)
        for k in range(1, 14):
            term = _mul(term, q / (4.0 * k))
            e = e + term
        e = _mul(e, e)
        out.append(_mul(_mul(e, e), u[mu]))
    return torch.stack(out)


def _loops(u):
    """c_plaq sum Re tr plaquettes + c_rect sum Re tr 2x1 rectangles."""
    total = 0.0
    for mu in range(4):
        for nu in range(4):
            if nu == mu:
                continue
            corner = _mul(u[nu], _to(u[mu], nu))                    # x -> x+nu -> x+nu+mu
            if nu > mu:
                total = total + C_PLAQ * _retr(_mul(u[mu], _to(u[nu], mu)), corner)
            two = _mul(u[mu], _to(u[mu], mu), _to(u[nu], mu, 2))    # x -> x+2mu -> x+2mu+nu
            total = total + C_RECT * _retr(two, _mul(corner, _to(_to(u[mu], mu), nu)))
    return total


def _retr(a, b):
    """Sum over sites of Re tr(a b^+)."""
    return (torch.view_as_real(a) * torch.view_as_real(b)).sum()


def _reals(f):
    return torch.view_as_real(f.resolve_conj().contiguous()).reshape(-1)


def exact(case, seed):
    gen = _gen(seed)
    kind, lat = case["kind"], _lat(case)
    u_lex = _links(case, gen)
    if kind == "smear":
        sigma = _su3(_algebra(case, gen), lat)
        u = _su3(u_lex, lat).clone().requires_grad_(True)
        s = u
        for _ in range(NSMEAR):
            s = torch.utils.checkpoint.checkpoint(_stout, s, use_reentrant=False)
        # d Re tr(sigma U_smeared) over the thin links: grad = force^+
        torch.view_as_real(s).mul(torch.view_as_real(sigma.mH.resolve_conj().contiguous())).sum().backward()
        force = -2.0 * _traceless(_mul(u.detach(), u.grad.mH))
        return [_reals(s.detach()), _reals(force)]
    if kind == "gauge":
        u = _su3(u_lex, lat).clone().requires_grad_(True)
        _loops(u).backward()
        force = (-BETA / 3.0) * _traceless(_mul(u.detach(), u.grad.mH))
        ip = _su3(_algebra(case, gen), lat) + EPS * force
        u0 = u.detach()
        t = u0
        for k in range(8, 0, -1):       # the update's order-8 Taylor recursion
            t = u0 + (EPS / k) * _mul(ip, t)
        r1 = t[..., 0, :] / torch.linalg.vector_norm(t[..., 0, :], dim=-1, keepdim=True)
        r2 = t[..., 1, :] - (r1.conj() * t[..., 1, :]).sum(-1, keepdim=True) * r1
        r2 = r2 / torch.linalg.vector_norm(r2, dim=-1, keepdim=True)
        t = torch.stack([r1, r2, torch.linalg.cross(r1, r2).conj()], -2)
        return [_reals(ip), _reals(t)]
    small = _vol(case) * case["ls"] <= 8 ** 4 * 16
    if kind in ("cg", "shiftcg", "richardson") and not small:
        return None                     # a plain torch solve would take minutes
    e = _Exact(case, u_lex)
    w = _spinor(case, gen)
    if kind == "mult" and case["mode"] == "Deo":
        # D_eo takes the field as odd, its dagger as even
        first = e.stored(e.half(e.deo(e.full(w, 1)), 0), case["prec"])
        return [first, e.stored(e.half(e.deo(e.full(w, 0), True), 1), case["prec"])]
    psi = e.full(w, 0)
    del w
    if kind == "mult":
        return [e.stored(e.half(e.mult(case["mode"], psi), 0), case["prec"])]
    if kind == "force":
        return [e.force(psi)]
    shifts = _shifts(case) if kind == "shiftcg" else [0.0]
    return [e.stored(e.half(e.solve(psi, float(s)), 0), "f64") for s in shifts]
