"""Material values that are not finite, in the kernel-level operator and in one stage of
the FP64 time step.  The predicted level is NaN or infinite exactly where the same sums in FP64 are, and elsewhere within the
rounding of two sums of 80 products (2 x 80 x 2^-53 < 2^-45 of the largest value).  A
subdomain that is the whole grid steps part by part; after its first part the two interior
planes next to a side can be read as a halo, so the planted point lies there.
"""
import ctypes as C

import numpy as np
import pytest

import sw4lite_gb300 as sg
from oracle import oracle as O
from tests.gpu_util import dev, host, smooth_fields, smooth_material

pytestmark = pytest.mark.gpu
SHAPE = (40, 17, 21)


@pytest.fixture(scope="module", autouse=True)
def _lib():
    sg.build()
    O.lib()


def _predicted(mat, u, um, dt, h):
    """Planes i = 1, 2 of the predicted level, (3, nz + 4, ny + 4, 2)."""
    nx, ny, nz = SHAPE
    g = sg.grid_desc(nx, ny, nz, h, bc=(2,) * 6, sg_gp=6)
    lib, ew = sg.lib(), C.c_void_p()
    sg.check(lib.sw4g_ew_create_subdomain(C.byref(g), 1, nx, 1, ny, None, C.byref(ew)))
    keep = [dev(a) for a in (*mat, u, um)]
    sg.check(lib.sw4g_ew_set_material(ew, *[a.data_ptr() for a in keep[:3]], 1))
    sg.check(lib.sw4g_ew_set_time_step(ew, dt, 0.0))
    sg.check(lib.sw4g_ew_set_fields(ew, keep[3].data_ptr(), keep[4].data_ptr(), 1))
    sg.check(lib.sw4g_ew_step_part(ew, 0))
    buf = dev(np.zeros(lib.sw4g_ew_halo_bytes(ew, 0) // 8))
    sg.check(lib.sw4g_ew_halo_pack(ew, 0, 0, buf.data_ptr()))
    out = host(buf).reshape(3, nz + 4, ny + 4, 2)
    sg.check(lib.sw4g_ew_destroy(ew))
    prof = []
    for ax, n in enumerate(SHAPE):
        arr = [np.zeros(n + 4) for _ in range(3)]
        sg.check(lib.sw4g_supergrid_profile(C.byref(g), ax, *[a.ctypes.data_as(sg._D) for a in arr]))
        prof.append(arr[1])
    return out, prof


@pytest.mark.parametrize("which", ["mu", "lambda"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("i", [1, 2, 4])
def test_predicted_level_is_not_finite_where_fp64_sums_are_not(which, bad, i):
    nx, ny, nz = SHAPE
    h = 0.05
    mat = smooth_material(nx, ny, nz, seed=2)
    dt = 0.3 * h / float(np.sqrt(np.max((4 * mat[1] + mat[2]) / mat[0])))
    mat[1 if which == "mu" else 2].reshape(nz + 4, ny + 4, nx + 4)[12, 9, i + 1] = bad
    u, um = smooth_fields(nx, ny, nz, seed=7)
    got, st = _predicted(mat, u, um, dt, h)
    lu = np.zeros_like(u)
    O.rhs4sg(1, (-1, nx + 2, -1, ny + 2, -1, nz + 2), nz, [0] * 6, lu, u, mat[1], mat[2], h, *st)
    want = (2 * u - um + dt * dt / np.tile(mat[0], 3) * lu).reshape(3, nz + 4, ny + 4, nx + 4)[..., 2:4]
    m = (slice(None), slice(2, -2), slice(2, -2))
    assert np.array_equal(np.isfinite(got[m]), np.isfinite(want[m]))
    ok = np.isfinite(want[m])
    assert np.max(np.abs(got[m] - want[m])[ok]) <= 2.0 ** -45 * np.max(np.abs(u))


@pytest.mark.parametrize("soa", [1, 0])
@pytest.mark.parametrize("bad", [np.nan, -np.inf])
def test_operator_lambda_not_finite(soa, bad):
    """The kernel-level operator: lambda enters all components at its own point and one
    component along each axis.  The bar is that of the operator's tile tests."""
    nx, ny, nz = SHAPE
    _, mu, la = smooth_material(nx, ny, nz, seed=4)
    u, _ = smooth_fields(nx, ny, nz, seed=5)
    la.reshape(nz + 4, ny + 4, nx + 4)[11, 8, 30] = bad
    st = [np.ones(n + 4) for n in SHAPE]
    b = (-1, nx + 2, -1, ny + 2, -1, nz + 2)
    want = np.zeros_like(u)
    O.rhs4sg(soa, b, nz, [0] * 6, want, u, mu, la, 0.3, *st)
    lu = dev(np.zeros_like(u))
    d = [dev(a) for a in (u, mu, la, *st)]
    sg.check(sg.lib().sw4g_rhs4sg(soa, *b, nz, (C.c_int * 6)(), lu.data_ptr(), *[t.data_ptr() for t in d[:3]], 0.3,
                                  *[t.data_ptr() for t in d[3:]], None))
    got = host(lu)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    ok = np.isfinite(want)
    scale = 64 * np.max((2 * mu + la)[np.isfinite(la)]) * np.max(np.abs(u)) / 0.3 ** 2
    assert np.max(np.abs(got - want)[ok]) <= 2.0 ** -46 * scale


@pytest.mark.parametrize("case", ["mu s", "(2 mu + lambda) s", "sx sy", "sx sz"])
def test_operator_products_that_overflow(case):
    """Finite inputs whose products are not: mu or 2 mu + lambda times a factor, or two factors
    of one point; the sums in FP64 are then infinite or NaN."""
    nx, ny, nz = SHAPE
    _, mu, la = smooth_material(nx, ny, nz, seed=4)
    u, _ = smooth_fields(nx, ny, nz, seed=5)
    st = [np.ones(n + 4) for n in SHAPE]
    if case == "mu s":
        mu *= 1e150
        la *= 1e-150
        st[1][9] = 1e200
    elif case == "(2 mu + lambda) s":
        la *= 1e150
        st[1][9] = 1e200
    else:
        mu *= 1e-200
        la *= 1e-200
        st[0][20] = 1e160
        st[1 if case == "sx sy" else 2][8] = -1e160
    b = (-1, nx + 2, -1, ny + 2, -1, nz + 2)
    want = np.zeros_like(u)
    O.rhs4sg(1, b, nz, [0] * 6, want, u, mu, la, 0.3, *st)
    lu = dev(np.zeros_like(u))
    d = [dev(a) for a in (u, mu, la, *st)]
    sg.check(sg.lib().sw4g_rhs4sg(1, *b, nz, (C.c_int * 6)(), lu.data_ptr(), *[t.data_ptr() for t in d[:3]], 0.3,
                                  *[t.data_ptr() for t in d[3:]], None))
    assert not np.all(np.isfinite(want))
    assert np.array_equal(np.isfinite(host(lu)), np.isfinite(want))


def test_ghost_edges_of_the_material_are_in_no_stencil():
    """Material that is NaN on the ghost points off two axes' interiors: the same bits as with
    finite values there."""
    nx, ny, nz = SHAPE
    mat = smooth_material(nx, ny, nz, seed=2)
    dt = 0.3 * 0.05 / float(np.sqrt(np.max((4 * mat[1] + mat[2]) / mat[0])))
    u, um = smooth_fields(nx, ny, nz, seed=7)
    want, _ = _predicted(mat, u, um, dt, 0.05)
    k, j, i = np.meshgrid(*[(np.arange(n + 4) < 2) | (np.arange(n + 4) >= n + 2) for n in (nz, ny, nx)], indexing="ij")
    edges = (i.astype(int) + j + k >= 2).ravel()
    for a in mat[1:]:
        a[edges] = np.nan
    got, _ = _predicted(mat, u, um, dt, 0.05)
    m = (slice(None), slice(2, -2), slice(2, -2))
    assert np.array_equal(got[m], want[m])
