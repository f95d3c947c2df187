"""Each component of a field, each axis and each coefficient keeps the digits that FP64 sums
give it: fields whose components differ by many powers of two, material whose coefficients
do, a displacement that is constant but for a small part, and stretching that falls to 1e-4.

Bars.  The predicted level is 2u - um + dt^2/rho L(u): three roundings on 2u - um and the
sum, six on the way from L(u) to it, and in L(u) a weight of five roundings, or a
coefficient of three, and a sum of 24 products: 2^-53 (3 (2|u| + |um|) + 16 dt^2/rho T) with
T the magnitudes that tests/wide.py sums.  Of fields that depend on one coordinate only, in
material that does not vary, the components are not coupled (the outer differences of equal
products are zero in any arithmetic): T is then that of the component by itself.  The
kernel-level operator is held to 2^-53 16 T with the second differences' magnitudes taken of
the differences of the values, which FP64 forms almost exactly.
"""
import ctypes as C

import numpy as np
import pytest

import sw4lite_gb300 as sg
from tests import wide
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu
SHAPE = (37, 21, 19)
H = 0.05


@pytest.fixture(scope="module", autouse=True)
def _lib():
    sg.build()


def _grid_arrays():
    nx, ny, nz = SHAPE
    return np.meshgrid(np.arange(nz + 4), np.arange(ny + 4), np.arange(nx + 4), indexing="ij")[::-1]


def _predict(mat, u, um, dt, sides):
    """The interior planes of the predicted level next to the four lateral sides, as
    (index, values) pairs into a (3, nk, nj, ni) array, and the stretching profiles."""
    nx, ny, nz = SHAPE
    g = sg.grid_desc(nx, ny, nz, H, bc=(sides,) * 6, sg_gp=6)
    lib, ew = sg.lib(), C.c_void_p()
    sg.check(lib.sw4g_ew_create_subdomain(C.byref(g), 1, nx, 1, ny, None, C.byref(ew)))
    keep = [dev(np.ascontiguousarray(a.ravel())) for a in (*mat, u, um)]
    sg.check(lib.sw4g_ew_set_material(ew, *[a.data_ptr() for a in keep[:3]], 1))
    sg.check(lib.sw4g_ew_set_time_step(ew, dt, 0.0))
    sg.check(lib.sw4g_ew_set_fields(ew, keep[3].data_ptr(), keep[4].data_ptr(), 1))
    sg.check(lib.sw4g_ew_step_part(ew, 0))
    out = []
    for axis in range(2):
        for side in range(2):
            n = SHAPE[axis]
            span = slice(2, 4) if side == 0 else slice(n, n + 2)
            where = (slice(None), slice(None), slice(None), span) if axis == 0 else (slice(None), slice(None), span)
            buf = dev(np.zeros(lib.sw4g_ew_halo_bytes(ew, axis) // 8))
            sg.check(lib.sw4g_ew_halo_pack(ew, axis, side, buf.data_ptr()))
            x = host(buf).reshape(3, nz + 4, (ny if axis == 0 else nx) + 4, 2)  # the two planes last
            out.append((where, x if axis == 0 else x.swapaxes(2, 3)))
    sg.check(lib.sw4g_ew_destroy(ew))
    st = []
    for ax, n in enumerate(SHAPE):
        arr = [np.ones(n + 4) for _ in range(3)]
        if sides == 2:
            sg.check(lib.sw4g_supergrid_profile(C.byref(g), ax, *[a.ctypes.data_as(sg._D) for a in arr]))
        st.append(arr[1])
    return out, st


def _check(mat, u, um, sides, coupled, least=0):
    rho, mu, la = mat
    dt = 0.3 * H / float(np.sqrt(np.max((4 * mu + la) / rho)))
    got, st = _predict(mat, u, um, dt, sides)
    val, terms = wide.operator(u, mu, la, st, H)
    if not coupled:
        for c in range(3):
            alone = np.zeros_like(u)
            alone[c] = u[c]
            terms[c] = wide.operator(alone, mu, la, st, H)[1][c]
    d2 = wide.L(dt) ** 2 / wide.L(1) / rho
    want = 2 * wide.L(1) * u - um + d2 * val
    bar = wide.L(2) ** -53 * (3 * (2 * abs(u) + abs(um)) + 16 * d2 * terms) + least
    for where, x in got:
        sel = (slice(None), slice(2, -2), slice(2, -2), slice(2, -2))
        full = np.full(u.shape, np.nan)
        full[where] = x
        err = np.abs(full[sel] - want[sel])
        ok = np.isfinite(full[sel])
        assert ok.any() and np.all(err[ok] <= bar[sel][ok]), float(np.max((err / bar[sel])[ok]))


def _material(rng, ratio=2.0, varying=True):
    x, y, z = _grid_arrays()
    f = 1 + (0.1 * np.sin(0.3 * x + 0.2 * y + 0.4 * z) if varying else 0 * x)
    return 2.0 * f, 1.3 * f, 1.3 * ratio * f


@pytest.mark.parametrize("sides", [1, 2])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", [10, 20, 40, 300])
def test_components_far_apart_in_plane_waves(sides, axis, n):
    rng = np.random.default_rng(n + axis)
    x = _grid_arrays()[axis]
    u, um = [np.stack([2.0 ** -(n * ((c - axis) % 3)) * np.sin(0.4 * x + rng.uniform(0, 6)) for c in range(3)])
             for _ in range(2)]
    _check(_material(rng, varying=False), u, um, sides, coupled=False)


@pytest.mark.parametrize("sides", [1, 2])
@pytest.mark.parametrize("scale", [(0, 20, 40), (60, 0, 30), (500, 700, 0)])
def test_components_far_apart_coupled(sides, scale):
    rng = np.random.default_rng(sum(scale))
    x, y, z = _grid_arrays()
    u, um = [np.stack([2.0 ** -scale[c] * np.sin(0.4 * x + rng.uniform(0, 6)) * np.cos(0.3 * y + rng.uniform(0, 6)) *
                       np.cos(0.5 * z + rng.uniform(0, 6)) for c in range(3)]) for _ in range(2)]
    _check(_material(rng), u, um, sides, coupled=True)


def _largest(rng, shape):
    return rng.choice([-1.0, 1.0], shape) * (2 - 2.0 ** -52)


@pytest.mark.parametrize("sides", [1, 2])
def test_largest_significands(sides):
    """Values of one magnitude with all bits set and signs at random: the largest integers that
    the sums meet."""
    rng = np.random.default_rng(sides)
    shape = (3,) + _grid_arrays()[0].shape
    mat = [np.full(shape[1:], 1.0), np.full(shape[1:], 2 - 2.0 ** -52), np.full(shape[1:], 4 - 2.0 ** -51)]
    _check(mat, _largest(rng, shape), _largest(rng, shape), sides, coupled=True)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", [15, 30, 45])
def test_constant_displacement_with_a_small_part(axis, n):
    """The differences of the large component are small: what they bring to the others is
    relative to the differences."""
    rng = np.random.default_rng(n)
    x, y, z = _grid_arrays()
    wave = np.stack([np.sin(0.4 * x + 0.3 * y + 0.2 * z + rng.uniform(0, 6)) for c in range(3)])
    u = 2.0 ** -n * wave
    u[axis] += 1.0
    _check(_material(rng), u, 0.9 * u, 1, coupled=True)


@pytest.mark.parametrize("sides", [1, 2])
@pytest.mark.parametrize("ratio", [30.0, 1e3, 1e9, 1e-9])
def test_soft_and_stiff_coefficients(sides, ratio):
    """mu and lambda apart: transverse waves, whose weights are mu's alone, and general ones."""
    rng = np.random.default_rng(5)
    x, y, z = _grid_arrays()
    u = np.zeros((3,) + x.shape)
    u[2] = np.sin(0.4 * x + 0.1)
    _check(_material(rng, ratio, varying=False), u, 0.8 * u, sides, coupled=False)
    u = np.stack([np.sin(0.4 * x + 0.3 * y - 0.2 * z + c) for c in range(3)])
    _check(_material(rng, ratio), u, 0.8 * u, sides, coupled=True)


def _check_operator(u, mu, la, st, coupled, soa, least=0):
    val, terms = wide.operator(u, mu, la, st, H, differences=True)
    if not coupled:
        for c in range(3):
            alone = np.zeros_like(u)
            alone[c] = u[c]
            terms[c] = wide.operator(alone, mu, la, st, H, differences=True)[1][c]
    nx, ny, nz = SHAPE
    b = (-1, nx + 2, -1, ny + 2, -1, nz + 2)
    lay = np.moveaxis(u, 0, 3) if not soa else u
    d = [dev(np.ascontiguousarray(a).ravel()) for a in (lay, mu, la, *st)]
    lu = dev(np.zeros(u.size))
    sg.check(sg.lib().sw4g_rhs4sg(soa, *b, nz, (C.c_int * 6)(), lu.data_ptr(), *[t.data_ptr() for t in d[:3]], H,
                                  *[t.data_ptr() for t in d[3:]], None))
    got = host(lu).reshape(u.shape) if soa else np.moveaxis(host(lu).reshape(*u.shape[1:], 3), 3, 0)
    sel = (slice(None), slice(2, -2), slice(2, -2), slice(2, -2))
    bar = 16 * wide.L(2) ** -53 * terms[sel] + least
    err = abs(got[sel] - val[sel])
    with np.errstate(all="ignore"):
        assert np.all(err <= bar), float(np.nanmax(np.where(bar > 0, err / bar, np.inf * err)))


def _profiles(kind, rng):
    st = []
    for n in SHAPE:
        s = np.ones(n + 4)
        if kind == "layers":
            s = np.maximum(1e-4, 1 - np.abs(np.linspace(-1, 1, n + 4)) ** 3)
        if kind == "any":
            s = rng.choice([-1.0, 1.0], n + 4) * np.ldexp(1 + rng.random(n + 4), rng.integers(-30, 30, n + 4))
            s[::9] = 0
        st.append(s)
    return st


@pytest.mark.parametrize("soa", [1, 0])
@pytest.mark.parametrize("profile", ["ones", "layers"])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", [10, 40, 300])
def test_operator_components_far_apart_in_plane_waves(soa, profile, axis, n):
    rng = np.random.default_rng(n + axis)
    x = _grid_arrays()[axis]
    u = np.stack([2.0 ** -(n * ((c - axis) % 3)) * np.sin(0.4 * x + rng.uniform(0, 6)) for c in range(3)])
    st = _profiles(profile, rng)
    if profile == "layers":  # equal products need equal factors along the other axes
        st = [s if a == axis else np.ones_like(s) for a, s in enumerate(st)]
    _, mu, la = _material(rng, varying=False)
    _check_operator(u, mu, la, st, False, soa)


@pytest.mark.parametrize("profile", ["ones", "layers", "any"])
@pytest.mark.parametrize("scale", [(0, 0, 0), (0, 20, 40), (500, 700, 0)])
@pytest.mark.parametrize("ratio", [2.0, 1e3, 1e-9])
def test_operator_coupled(profile, scale, ratio):
    rng = np.random.default_rng(sum(scale))
    x, y, z = _grid_arrays()
    u = np.stack([2.0 ** -scale[c] * np.sin(0.4 * x + rng.uniform(0, 6)) * np.cos(0.3 * y + rng.uniform(0, 6)) *
                  np.cos(0.5 * z + rng.uniform(0, 6)) for c in range(3)])
    _, mu, la = _material(rng, ratio)
    _check_operator(u, mu, la, _profiles(profile, rng), True, 1)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", [15, 30, 45])
def test_operator_constant_displacement_with_a_small_part(axis, n):
    rng = np.random.default_rng(n)
    x, y, z = _grid_arrays()
    u = np.stack([2.0 ** -n * np.sin(0.4 * x + 0.3 * y + 0.2 * z + rng.uniform(0, 6)) for c in range(3)])
    u[axis] += 1.0
    _, mu, la = _material(rng)
    _check_operator(u, mu, la, _profiles("ones", rng), True, 1)


@pytest.mark.parametrize("profile", ["ones", "layers", "any"])
def test_operator_largest_significands(profile):
    rng = np.random.default_rng(8)
    u = _largest(rng, (3,) + _grid_arrays()[0].shape)
    mu, la = [f * np.ones(u.shape[1:]) for f in (2 - 2.0 ** -52, 4 - 2.0 ** -51)]
    _check_operator(u, mu, la, _profiles(profile, rng), True, 1)
    la *= -1  # coefficients of both signs
    mu *= np.where(_grid_arrays()[0] % 2 == 0, 1.0, -1.0)
    _check_operator(u, mu, la, _profiles(profile, rng), True, 1)


LEAST = wide.L(2) ** -1074


@pytest.mark.skipif(LEAST / 4 == 0, reason="needs an extended exponent range")
def test_below_the_normal_range():
    """Levels and results below 2^-1022 are rounded to multiples of 2^-1074, as FP64 does it: the
    sum, the product dt^2/rho L and L itself, each once (half a unit), dt^2/rho being below 1.
    The operator rounds its sum and the product with 1/(144 h^2) = 2.8, which multiplies the
    first's half unit."""
    rng = np.random.default_rng(3)
    x, y, z = _grid_arrays()
    wave = np.stack([np.sin(0.4 * x + 0.3 * y + 0.5 * z + rng.uniform(0, 6)) for c in range(3)])
    u = np.round(wave * 2 ** 14) * 2.0 ** -1074
    _check(_material(rng), u, 0.5 * np.round(u / 2.0 ** -1073) * 2.0 ** -1073, 2, True, least=2 * LEAST)
    _, mu, la = _material(rng)
    _check_operator(wave * 2.0 ** -440, mu * 2.0 ** -600, la * 2.0 ** -600, _profiles("layers", rng), True, 1, least=2 * LEAST)


@pytest.mark.skipif(LEAST / 4 == 0, reason="needs an extended exponent range")
def test_operator_factor_below_the_normal_range():
    """A stretching factor of 3 x 2^-1040 along x and coefficients of 2^900: the x component of a
    field in y has the mixed terms alone."""
    rng = np.random.default_rng(4)
    x, y, z = _grid_arrays()
    u = np.zeros((3,) + x.shape)
    u[1] = np.sin(0.4 * x + 0.3 * y + 0.5 * z)
    _, mu, la = _material(rng)
    st = _profiles("ones", rng)
    st[0][:] = 3 * 2.0 ** -1040
    _check_operator(u, mu * 2.0 ** 900, la * 2.0 ** 900, st, True, 1)
