"""The fixed-point stage kernels of the FP64 time step (csrc/stage_fixed.cu) where their
arithmetic and tiling can go wrong: extents at the edges of the 32 x 6 column tiles and
of the plane chunks, levels whose exponents span most of FP64's range within a few
points, zero and non-finite values, and the FP64 stages that take over where the device
has no room for the fixed-point coefficients.

Tolerance of one step from given levels: both sides evaluate, twice in a row, sums of
about 80 products of a material weight and a level, each within a few 2^-53 of its
largest term.  With the time step at 0.3 of the grid spacing over the largest speed the
weights' absolute sum times dt^2/rho is below 1, so the two differ at a point by less
than 2 x 80 x 2^-53 < 2^-45 of the largest value within the two operators' reach (four
points along each axis).
"""
import numpy as np
import pytest

import sw4lite_gb300 as sg
from oracle import oracle as O
from tests.gpu_util import OracleProblem, dev, host, smooth_fields, smooth_material

pytestmark = pytest.mark.gpu
H = 0.05


@pytest.fixture(scope="module", autouse=True)
def _lib():
    sg.build()
    O.lib()


def _step(g, mat, u, um, dt, nsteps=1):
    ew = sg.EW(g)
    ew.set_material(*[dev(a) for a in mat])
    ew.set_time_step(dt, 0.0)
    ew.set_fields(dev(u), dev(um))
    ew.step(nsteps)
    out = dev(np.zeros_like(u))
    ew.get_fields(out, None)
    r = host(out)
    ew.close()
    return r


def _problem(shape, top, seed=3, gp=6):
    nx, ny, nz = shape
    g = sg.grid_desc(nx, ny, nz, H, bc=(2, 2, 2, 2, top, 2), sg_gp=gp)
    mat = smooth_material(nx, ny, nz, seed=seed)
    dt = 0.3 * H / float(np.sqrt(np.max((4 * mat[1] + mat[2]) / mat[0])))
    return g, mat, dt


def _reach(u, shape):
    """The largest magnitude over all components within four points along each axis."""
    nx, ny, nz = shape
    a = np.abs(u.reshape(3, nz + 4, ny + 4, nx + 4)).max(axis=0)
    for ax in range(3):
        a = np.max([np.roll(a, m, axis=ax) for m in range(-4, 5)], axis=0)
    return np.broadcast_to(a, (3,) + a.shape).ravel()


def _check(g, mat, u, um, dt, shape):
    got = _step(g, mat, u, um, dt)
    ref, _ = OracleProblem(g, *mat, dt, ()).run(u, um, 0.0, 1)
    bound = 2.0 ** -45 * np.maximum(_reach(u, shape), _reach(um, shape))
    assert np.all(np.abs(got - ref) <= bound + 1e-300)


@pytest.mark.parametrize("shape", [(8, 8, 8), (31, 5, 9), (32, 6, 14), (33, 7, 15), (34, 12, 25), (63, 13, 27),
                                   (65, 17, 53)])
@pytest.mark.parametrize("top", [2, 0])
def test_tile_edges(shape, top):
    if top == 0 and shape[2] < 14:
        pytest.skip("a free surface needs 14 planes")
    if shape[1] < 8:
        shape = (shape[0], shape[1] + 6, shape[2])
    if shape[2] < 8:
        shape = shape[:2] + (8,)
    g, mat, dt = _problem(shape, top, gp=3)
    _check(g, mat, *smooth_fields(*shape, seed=5), dt, shape)


@pytest.mark.parametrize("span", [40, 300, 1000])
def test_exponents_far_apart(span):
    """Random signs, exponents random between 0 and -span at every point, and a wedge of
    zeros."""
    shape = (36, 14, 20)
    g, mat, dt = _problem(shape, 2)
    rng = np.random.default_rng(span)
    n = mat[0].size
    u, um = [rng.choice([-1.0, 1.0], 3 * n) * np.ldexp(1.0 + rng.random(3 * n), rng.integers(-span, 1, 3 * n))
             for _ in range(2)]
    for a in (u, um):
        a.reshape(3, 24, 18, 40)[:, :, :, 25:] = 0
    _check(g, mat, u, um, dt, shape)


def test_smooth_decay_keeps_relative_accuracy():
    """Levels that fall by 2^-20 a point: the bound above is local, so the small values
    keep their digits."""
    shape = (40, 12, 16)
    g, mat, dt = _problem(shape, 2)
    i = np.arange(44)
    base = np.ldexp(1.0, -20 * i)
    rng = np.random.default_rng(4)
    u, um = [(base * (1 + rng.random((3, 20, 16, 44)))).ravel() for _ in range(2)]
    _check(g, mat, u, um, dt, shape)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_values_reach_the_stencil_and_no_further(bad):
    shape = (40, 20, 24)
    g, mat, dt = _problem(shape, 2)
    u, um = smooth_fields(*shape, seed=9)
    u.reshape(3, 28, 24, 44)[2, 13, 11, 21] = bad
    got = _step(g, mat, u, um, dt)
    ref, _ = OracleProblem(g, *mat, dt, ()).run(u, um, 0.0, 1)
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))


@pytest.mark.parametrize("order", [4, 6])
@pytest.mark.parametrize("shape,gp,top", [((190, 180, 176), 30, 0), ((61, 44, 40), 6, 2), ((40, 36, 38), 25, 2)])
def test_damping_of_the_layers(order, shape, gp, top):
    """The layers' own kernel (fused steps) against the kernel that visits every point
    (the phase order): long and short marches, layers on both sides of an axis and
    layers that meet, edges and corners in two and three layers."""
    nx, ny, nz = shape
    g = sg.grid_desc(nx, ny, nz, H, bc=(2, 2, 2, 2, top, 2), sg_gp=gp, sg_damping=0.02, sg_order=order)
    _, mat, dt = _problem(shape, top)
    u, um = smooth_fields(*shape, seed=8)
    out = []
    for mode in (sg.MODE_FUSED, sg.MODE_PHASES):
        ew = sg.EW(g)
        ew.set_material(*[dev(a) for a in mat])
        ew.set_time_step(dt, 0.0)
        ew.set_fields(dev(u), dev(um))
        ew.step(1, mode)
        r = dev(np.zeros_like(u))
        ew.get_fields(r, None)
        out.append(host(r))
        ew.close()
    assert np.max(np.abs(out[0] - out[1])) <= 2.0 ** -45 * np.max(np.abs(out[1]))


def test_without_room_for_the_coefficients_the_fp64_stages_run():
    import torch
    shape = (200, 180, 160)
    g, mat, dt = _problem(shape, 0, gp=15)
    u, um = smooth_fields(*shape, seed=2)
    n = mat[0].size
    torch.cuda.empty_cache()

    def run():
        before = torch.cuda.mem_get_info()[0]
        ew = sg.EW(g)
        used = before - torch.cuda.mem_get_info()[0]
        ew.set_material(*mat)
        ew.set_time_step(dt, 0.0)
        ew.set_fields(u, um)
        ew.step(3)
        out = np.zeros_like(u)
        ew.get_fields(out, None)
        ew.close()
        return out, used / n

    roomy, used = run()
    assert used > 330
    # leave room for the object with the FP64 weights (272 bytes a point), not for more
    fill = torch.empty(torch.cuda.mem_get_info()[0] - 330 * n, dtype=torch.uint8, device="cuda")
    tight, used = run()
    del fill
    torch.cuda.empty_cache()
    assert 260 < used < 300
    assert np.max(np.abs(tight - roomy)) <= 1e-13 * np.max(np.abs(roomy))
