"""Kernel-level parity on the GPU: each C-ABI kernel entry point against the CPU
oracle (oracle/sw4_oracle.c) on seeded random fields.

Tolerances (FP64): the operator and damping kernels agree with the oracle to
1e-13 relative to the largest output magnitude (different summation order and
FMA contraction); pointwise updates and ghost copies to 1e-14.
"""
import ctypes as C

import numpy as np
import pytest

import sw4lite_gb300 as sg
from oracle import oracle as O
from tests.fields import Grid, rel_err
from tests.gpu_util import dev, host, stream

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    sg.build()
    O.lib()


def _onesided(t, b):
    a = (C.c_int * 6)()
    a[4], a[5] = t, b
    return a


@pytest.mark.parametrize("soa", [1, 0])
@pytest.mark.parametrize("onesided", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("shape", [(13, 11, 17), (40, 9, 21), (33, 29, 27)])
def test_rhs4sg(soa, onesided, shape):
    g = Grid(*shape, h=0.37)
    rng = np.random.default_rng(11 + soa + 3 * onesided[0] + 5 * onesided[1])
    u = g.field3(rng)
    rho, mu, la = g.material(rng)
    sx, sy, sz = g.stretching(rng)
    os6 = [0, 0, 0, 0, onesided[0], onesided[1]]
    ref = np.zeros_like(u)
    O.rhs4sg(soa, g.bounds, g.nz, os6, ref, u, mu, la, g.h, sx, sy, sz)
    du, dmu, dla, dsx, dsy, dsz = (dev(a) for a in (u, mu, la, sx, sy, sz))
    dlu = dev(np.zeros_like(u))
    st = sg.lib().sw4g_rhs4sg(soa, *g.bounds, g.nz, _onesided(*onesided), dlu.data_ptr(),
                              du.data_ptr(), dmu.data_ptr(), dla.data_ptr(), g.h, dsx.data_ptr(),
                              dsy.data_ptr(), dsz.data_ptr(), stream())
    sg.check(st, "sw4g_rhs4sg")
    got = host(dlu)
    assert rel_err(got, ref) <= 1e-13
    # ghost shell untouched
    m = g.interior_mask()
    assert np.all(g.as4(got, soa)[:, ~m] == 0)


@pytest.mark.parametrize("soa", [1, 0])
def test_pointwise_updates(soa):
    g = Grid(17, 12, 10)
    rng = np.random.default_rng(3 + soa)
    up0, u, um, lu, fo = (g.field3(rng) for _ in range(5))
    rho, _, _ = g.material(rng)
    dt = 0.0123
    L = sg.lib()
    d = {k: dev(v) for k, v in dict(up=up0, u=u, um=um, lu=lu, fo=fo, rho=rho).items()}
    # predictor
    ref = up0.copy()
    O.predfort(soa, g.bounds, ref, u, um, lu, fo, rho, dt * dt)
    sg.check(L.sw4g_predfort(soa, *g.bounds, d["up"].data_ptr(), d["u"].data_ptr(),
                             d["um"].data_ptr(), d["lu"].data_ptr(), d["fo"].data_ptr(),
                             d["rho"].data_ptr(), dt * dt, stream()))
    np.testing.assert_allclose(host(d["up"]), ref, rtol=1e-14, atol=1e-15)
    # corrector on top of it
    O.corrfort(soa, g.bounds, ref, lu, fo, rho, dt ** 4)
    sg.check(L.sw4g_corrfort(soa, *g.bounds, d["up"].data_ptr(), d["lu"].data_ptr(),
                             d["fo"].data_ptr(), d["rho"].data_ptr(), dt ** 4, stream()))
    np.testing.assert_allclose(host(d["up"]), ref, rtol=1e-14, atol=1e-15)
    # dpdm
    ref2 = np.zeros_like(u)
    O.dpdmtfort(g.bounds, up0, u, um, ref2, 1 / dt ** 2)
    out = dev(np.zeros_like(u))
    dup0 = dev(up0)
    sg.check(L.sw4g_dpdmtfort(*g.bounds, dup0.data_ptr(), d["u"].data_ptr(),
                              d["um"].data_ptr(), out.data_ptr(), 1 / dt ** 2, stream()))
    np.testing.assert_allclose(host(out), ref2, rtol=1e-14, atol=1e-12)


@pytest.mark.parametrize("order", [4, 6])
@pytest.mark.parametrize("soa", [1, 0])
def test_addsgd(order, soa):
    g = Grid(19, 14, 16)
    rng = np.random.default_rng(21 + order + soa)
    up0, u, um = g.field3(rng), g.field3(rng), g.field3(rng)
    rho, _, _ = g.material(rng)
    dc = (g.strip(rng, g.ni, 0, 1), g.strip(rng, g.nj, 0, 1), g.strip(rng, g.nk, 0, 1))
    st = g.stretching(rng)
    co = (g.strip(rng, g.ni, 0.3, 1), g.strip(rng, g.nj, 0.3, 1), g.strip(rng, g.nk, 0.3, 1))
    ref = up0.copy()
    O.addsgd(order, soa, g.bounds, ref, u, um, rho, dc, st, co, 0.02)
    # every device buffer stays referenced until the kernel has run
    dup, du, dum, drho = dev(up0), dev(u), dev(um), dev(rho)
    prof = [dev(a) for a in (*dc, *st, *co)]
    fn = sg.lib().sw4g_addsgd6fort if order == 6 else sg.lib().sw4g_addsgd4fort
    sg.check(fn(soa, *g.bounds, dup.data_ptr(), du.data_ptr(), dum.data_ptr(),
                drho.data_ptr(), *[p.data_ptr() for p in prof], 0.02, stream()))
    got = host(dup)
    assert rel_err(got - up0, ref - up0) <= 1e-13


@pytest.mark.parametrize("soa", [1, 0])
@pytest.mark.parametrize("bccnd", [(2, 2, 2, 2, 0, 2), (1, 1, 1, 1, 1, 1), (3, 3, 3, 3, 0, 0),
                                   (2, 2, 2, 2, 2, 0)])
def test_bcfortsg(soa, bccnd):
    g = Grid(15, 13, 12, h=0.5)
    rng = np.random.default_rng(31 + soa)
    u0 = g.field3(rng)
    _, mu, la = g.material(rng)
    sx, sy, _ = g.stretching(rng)
    wind, npts = O.boundary_windows(g.bounds, (g.nx, g.ny, g.nz), bccnd)
    bforce = [g.field3(rng)[: 3 * max(1, n)].copy() if bccnd[s] in (0, 1) else None
              for s, n in enumerate(npts)]
    _, _, _, sbop = O.stencil_coefficients()
    ref = u0.copy()
    O.bcfortsg(soa, g.bounds, wind, (g.nx, g.ny, g.nz), ref, g.h, bccnd, sbop, mu, la, bforce, sx, sy)
    du = dev(u0)
    dbf = [dev(b) if b is not None else None for b in bforce]
    ptrs = (C.c_void_p * 6)(*[b.data_ptr() if b is not None else None for b in dbf])
    w = (C.c_int * 36)(*[int(x) for x in wind])
    bc = (C.c_int * 6)(*bccnd)
    sb = (C.c_double * 6)(*sbop)
    dmu, dla, dsx, dsy = dev(mu), dev(la), dev(sx), dev(sy)
    sg.check(sg.lib().sw4g_bcfortsg(soa, *g.bounds, w, g.nx, g.ny, g.nz, du.data_ptr(), g.h, bc,
                                    C.cast(sb, sg._D), dmu.data_ptr(), dla.data_ptr(), ptrs,
                                    dsx.data_ptr(), dsy.data_ptr(), stream()))
    assert rel_err(host(du), ref) <= 1e-14


def _operator(g, soa, u, mu, la, st):
    lu = dev(np.zeros_like(u))
    d = [dev(a) for a in (u, mu, la, *st)]
    sg.check(sg.lib().sw4g_rhs4sg(soa, *g.bounds, g.nz, _onesided(0, 0), lu.data_ptr(), d[0].data_ptr(), d[1].data_ptr(),
                                  d[2].data_ptr(), g.h, *[t.data_ptr() for t in d[3:]], stream()))
    return host(lu)


@pytest.mark.parametrize("soa", [1, 0])
@pytest.mark.parametrize("shape", [(1, 1, 1), (31, 5, 3), (32, 6, 2), (33, 7, 41), (65, 13, 14)])
@pytest.mark.parametrize("profile", ["ones", "layers", "any"])
def test_operator_tiles_and_profiles(soa, shape, profile):
    """Extents at the edges of the operator's 32 x 6 column tiles and of its marches, and
    stretching profiles of 1, falling to 1e-4 at the sides, and of any sign and size with
    zeros.  Both sides form sums of about 80 products, each within a few 2^-53 of the
    largest, (2 mu + lambda) |s|^2 |u| / h^2 times weights that add to less than 64: they
    differ by less than 2^-46 of 64 such terms."""
    g = Grid(*shape, h=0.37)
    rng = np.random.default_rng(sum(shape) + soa)
    u = g.field3(rng)
    _, mu, la = g.material(rng, spread=0.9)
    st = []
    for n in (g.ni, g.nj, g.nk):
        s = np.ones(n)
        if profile == "layers":
            s = np.maximum(1e-4, np.minimum(1, (np.abs(np.arange(n) - n / 2) / (n / 2) - 1) ** 2))
        if profile == "any":
            s = rng.choice([-1.0, 1.0], n) * np.ldexp(1 + rng.random(n), rng.integers(-30, 30, n))
            s[:: max(2, n // 3)] = 0
        st.append(np.ascontiguousarray(s))
    ref = np.zeros_like(u)
    O.rhs4sg(soa, g.bounds, g.nz, [0] * 6, ref, u, mu, la, g.h, *st)
    got = _operator(g, soa, u, mu, la, st)
    big = max(np.max(np.abs(s)) for s in st)
    scale = 64 * np.max(2 * mu + la) * big * big * np.max(np.abs(u)) / g.h ** 2
    assert np.max(np.abs(got - ref)) <= 2.0 ** -46 * scale


@pytest.mark.parametrize("where", ["u", "mu", "sz"])
def test_operator_non_finite_inputs(where):
    g = Grid(40, 20, 22, h=0.3)
    rng = np.random.default_rng(3)
    u = g.field3(rng)
    _, mu, la = g.material(rng)
    st = list(g.stretching(rng))
    if where == "u":
        u.reshape(3, g.nk, g.nj, g.ni)[1, 12, 9, 20] = np.inf
    elif where == "mu":
        mu.reshape(g.nk, g.nj, g.ni)[12, 9, 20] = np.nan
    else:
        st[2][11] = np.nan
    ref = np.zeros_like(u)
    O.rhs4sg(1, g.bounds, g.nz, [0] * 6, ref, u, mu, la, g.h, *st)
    assert np.array_equal(np.isfinite(_operator(g, 1, u, mu, la, st)), np.isfinite(ref))


@pytest.mark.parametrize("soa", [1, 0])
@pytest.mark.parametrize("nz,planes", [(3, None), (12, (3, 6)), (12, (-1, 0))])
def test_bcfortsg_zero_window_among_the_free_surface_planes(soa, nz, planes):
    """The window of side 5 meets the planes that the free surface on side 4 reads or writes: a
    grid of three planes, and a caller's own window.  The sides act in their order."""
    bccnd = (2, 2, 2, 2, 0, 2)
    g = Grid(15, 13, nz, h=0.5)
    rng = np.random.default_rng(7 + soa)
    u0 = g.field3(rng)
    _, mu, la = g.material(rng)
    sx, sy, _ = g.stretching(rng)
    wind, _ = O.boundary_windows(g.bounds, (g.nx, g.ny, g.nz), bccnd)
    wind = [int(x) for x in wind]
    if planes:
        wind[34:36] = planes
    _, _, _, sbop = O.stencil_coefficients()
    ref = u0.copy()
    O.bcfortsg(soa, g.bounds, wind, (g.nx, g.ny, g.nz), ref, g.h, bccnd, sbop, mu, la, [None] * 6, sx, sy)
    du, dmu, dla, dsx, dsy = dev(u0), dev(mu), dev(la), dev(sx), dev(sy)

    def sides(field, active):
        sg.check(sg.lib().sw4g_bcfortsg(soa, *g.bounds, (C.c_int * 36)(*wind), g.nx, g.ny, g.nz, field.data_ptr(), g.h,
                                        (C.c_int * 6)(*[b if s in active else 4 for s, b in enumerate(bccnd)]),
                                        C.cast((C.c_double * 6)(*sbop), sg._D), dmu.data_ptr(), dla.data_ptr(),
                                        (C.c_void_p * 6)(), dsx.data_ptr(), dsy.data_ptr(), stream()))

    one_by_one = dev(u0)
    for s in range(6):
        sides(one_by_one, (s,))
    sides(du, range(6))
    assert np.array_equal(host(du), host(one_by_one))
    assert rel_err(host(du), ref) <= 1e-14
