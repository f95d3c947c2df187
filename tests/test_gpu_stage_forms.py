"""The two forms of the FP64 stages (EW.stage_form): the FP64 one on the cases of the other
test modules, with their bars; changing the form; and the FP64 form taken where the
device has no room for the fixed-point one's coefficients.

Two runs of one problem in the two forms are each held to the oracle in those modules; here
they are compared with each other at the bar of one step between a form and the oracle
(tests/test_gpu_stage_fixed.py: 2^-45 of the largest value), times the steps.
"""
import numpy as np
import pytest

import sw4lite_gb300 as sg
from oracle import oracle as O
from tests import (wide, test_gpu_adjoint, test_gpu_graphs, test_gpu_halo, test_gpu_nancheck, test_gpu_stage_fixed,
                   test_gpu_step, test_gpu_topo)
from tests.adjoint_util import AdjointCase, oracle_forward
from tests.gpu_util import dev, host, smooth_fields, smooth_material

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    sg.build()
    O.lib()


@pytest.fixture
def fp64_form(monkeypatch):
    """Every FP64 object is changed to the FP64 stages when it is made."""
    made = []
    init = sg.EW.__init__

    def make(self, *args, **kw):
        init(self, *args, **kw)
        if self.stage_form() == sg.STAGES_FIXED:
            self.set_stage_form(sg.STAGES_FP64)
            made.append(self)

    monkeypatch.setattr(sg.EW, "__init__", make)
    yield
    assert made


@pytest.mark.parametrize("shape", [(8, 8, 8), (31, 9, 9), (32, 8, 14), (33, 15, 15), (65, 17, 53)])
@pytest.mark.parametrize("top", [2, 0])
def test_tile_edges(fp64_form, shape, top):
    if top == 0 and shape[2] < 14:
        shape = shape[:2] + (14,)
    g, mat, dt = test_gpu_stage_fixed._problem(shape, top, gp=3)
    test_gpu_stage_fixed._check(g, mat, *smooth_fields(*shape, seed=5), dt, shape)


@pytest.mark.parametrize("order", [4, 6])
def test_damping(fp64_form, order):
    test_gpu_stage_fixed.test_damping_of_the_layers(order, (61, 44, 40), 6, 2)


def test_non_finite_values(fp64_form):
    test_gpu_stage_fixed.test_non_finite_values_reach_the_stencil_and_no_further(np.nan)


@pytest.mark.parametrize("px,py", [(2, 1), (2, 2)])
def test_subdomains(fp64_form, px, py):
    assert test_gpu_halo._decomposed(px, py, 40, 36, 26, sg.FP64, 8) == 0


@pytest.mark.parametrize("ckpt,memory", [(30, None), (7, 0)])
def test_gradient(fp64_form, ckpt, memory):
    test_gpu_adjoint.test_gradient_matches_oracle_adjoint(ckpt, memory)


def test_graphs(fp64_form):
    test_gpu_graphs.test_graphed_steps_bit_identical(sg.FP64)


def test_steps(fp64_form):
    test_gpu_step.test_sixth_order_damping_step()
    test_gpu_step.test_fused_and_phase_paths_agree_over_many_steps()


def test_topography(fp64_form):
    test_gpu_topo.test_topo_steps_with_curvilinear_sources(sg.MODE_FUSED)


def _object(shape=(160, 150, 140), top=0):
    nx, ny, nz = shape
    g, mat, dt = test_gpu_stage_fixed._problem(shape, top, gp=15)
    ew = sg.EW(g)
    ew.set_material(*[dev(a) for a in mat])
    ew.set_time_step(dt, 0.0)
    return ew, smooth_fields(nx, ny, nz, seed=2)


def _steps(ew, u, um, n):
    ew.set_fields(dev(u), dev(um))
    ew.step(n)
    out = dev(np.zeros_like(u))
    ew.get_fields(out, None)
    return host(out)


def test_changing_the_form():
    import torch
    ew, (u, um) = _object()
    assert ew.stage_form() == sg.STAGES_FIXED
    fixed = _steps(ew, u, um, 2)
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    ew.set_stage_form(sg.STAGES_FP64)
    assert ew.stage_form() == sg.STAGES_FP64
    # 192 bytes an interior point and 32 an array point against 144 (allocations are rounded up)
    less = 192 * 160 * 150 * 140 - 112 * ew.npts
    assert torch.cuda.mem_get_info()[0] - free > less - (8 << 20)
    fp64 = _steps(ew, u, um, 2)
    assert np.max(np.abs(fp64 - fixed)) <= 2 * 2.0 ** -45 * np.max(np.abs(u))
    ew.set_stage_form(sg.STAGES_FIXED)
    assert np.array_equal(_steps(ew, u, um, 2), fixed)
    with pytest.raises(sg.Sw4gError):
        ew.set_stage_form(2)
    ew.close()


def test_the_mixed_form_has_no_choice():
    ew = sg.EW(sg.grid_desc(20, 20, 20, 0.1, sg_gp=5, precision=sg.MIXED))
    assert ew.stage_form() == -1
    with pytest.raises(sg.Sw4gError):
        ew.set_stage_form(sg.STAGES_FP64)
    ew.close()


def test_not_within_a_step():
    g = test_gpu_stage_fixed._problem((20, 20, 20), 2)[0]
    ew = sg.EW(g, subdomain=(1, 20, 1, 20))
    ew.set_material(*[dev(a) for a in smooth_material(20, 20, 20, seed=1)])
    ew.set_time_step(1e-3, 0.0)
    ew.step_part(0)
    with pytest.raises(sg.Sw4gError):
        ew.set_stage_form(sg.STAGES_FP64)
    ew.step_part(1)
    ew.step_part(2)
    ew.set_stage_form(sg.STAGES_FP64)
    ew.close()


def test_a_group_of_subdomains_steps_in_one_form():
    g, mat, fields, _, dt = test_gpu_halo._problem(40, 36, 26, sg.FP64)
    subs = []
    for i0, i1 in ((1, 20), (21, 40)):
        e = sg.EW(g, subdomain=(i0, i1, 1, 36))
        e.set_material(*[dev(test_gpu_halo._local(a, 40, 36, 26, i0, i1, 1, 36, 1)) for a in mat])
        e.set_time_step(dt, 0.0)
        e.set_fields(*[dev(test_gpu_halo._local(a, 40, 36, 26, i0, i1, 1, 36, 3)) for a in fields])
        subs.append(e)
    subs[1].set_stage_form(sg.STAGES_FP64)
    sg.step_group(subs, [[-1, 1, -1, -1], [0, -1, -1, -1]], 2)
    assert [e.stage_form() for e in subs] == [sg.STAGES_FP64] * 2
    for e in subs:
        e.close()


def _leave(free_bytes):
    import torch
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - free_bytes, dtype=torch.uint8, device="cuda")


def test_a_gradient_takes_the_room_of_the_coefficients():
    import torch
    ew, (u, um) = _object(top=2)
    n, steps = ew.npts, 3
    rec = [(40, 50, 60), (100, 70, 30)]
    ew.set_receivers(rec, [sg.REC_DISPLACEMENT] * 2, steps + 2)
    obs = np.zeros((steps + 1, 6))
    g = [dev(np.zeros(n)) for _ in range(3)]
    du, dum, dobs = dev(u), dev(um), dev(obs)

    def gradient():
        ew.set_time_step(1e-3, 0.0)
        ew.set_fields(du, dum)
        return ew.gradient(steps, steps, dobs, *g), [host(a) for a in g]

    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    misfit, want = gradient()
    takes = before - torch.cuda.mem_get_info()[0]
    assert ew.stage_form() == sg.STAGES_FIXED and takes > 100 * n
    ew.set_gradient_memory(0)  # gives its buffers back
    fill = _leave(takes - 40 * n)
    got_misfit, got = gradient()
    del fill
    torch.cuda.empty_cache()
    assert ew.stage_form() == sg.STAGES_FP64
    assert got_misfit == pytest.approx(misfit, rel=1e-12)
    for a, b in zip(got, want):
        assert np.max(np.abs(a - b)) <= 1e-9 * np.max(np.abs(b))
    # nothing is left of the refused allocation
    ew.step(1)
    ew.close()


def test_topography_takes_the_room_of_the_coefficients():
    """The curvilinear coefficients, allocated with its material, on a device that was filled
    since the object was made."""
    import torch
    from tests.topo_util import TopoCase
    c = TopoCase(150, 140, 120, 0.1, zmax_topo=1.0, amp=0.2, xc=7.0, yc=7.0, lx=2.0, ly=2.0, gp=15)

    def run(tight):
        ew = sg.EW(c.grid, topo=sg.topo_desc(**c.hill))
        ew.set_material(*[dev(a) for a in c.cart_mat])
        curv = [dev(a) for a in c.curv_mat]
        fill = _leave(30 << 20) if tight else None
        ew.set_material_grid(1, *curv)
        form = ew.stage_form()
        del fill
        torch.cuda.empty_cache()
        ew.set_time_step(1e-2, 0.0)
        x = np.sin(np.arange(3 * ew.npts) * 0.01)
        n1 = ew.grid_dims(1)[3]
        y = np.sin(np.arange(3 * n1) * 0.01)
        ew.set_fields(dev(x), dev(0.9 * x))
        ew.set_fields_grid(1, dev(y), dev(0.9 * y))
        ew.step(1)
        out = dev(np.zeros(3 * ew.npts))
        ew.get_fields(out, None)
        r = host(out)
        ew.close()
        return r, form

    a, form = run(False)
    assert form == sg.STAGES_FIXED
    b, form = run(True)
    assert form == sg.STAGES_FP64
    assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(a))


def test_the_fixed_form_is_no_further_off_than_fp64_sums():
    """Eight steps of both forms against extended precision (predictor, corrector, no damping):
    the error of the fixed-point form, over all components, is no larger."""
    nx, ny, nz = shape = (21, 20, 19)
    h, steps = 0.05, 8
    rho, mu, la = mat = smooth_material(nx, ny, nz, seed=6)
    dt = 0.3 * h / float(np.sqrt(np.max((4 * mu + la) / rho)))
    fields = smooth_fields(nx, ny, nz, seed=4, scale=1.0)
    cut = (slice(None),) + (slice(2, -2),) * 3
    for a in fields:  # ghost planes as a Dirichlet side leaves them
        b = a.reshape(3, nz + 4, ny + 4, nx + 4)
        inner = b[cut].copy()
        b[:] = 0
        b[cut] = inner
    u, um = [a.reshape(3, nz + 4, ny + 4, nx + 4).astype(wide.L) for a in fields]
    r, m, l = [a.reshape(nz + 4, ny + 4, nx + 4) for a in mat]
    one = [np.ones(n + 4) for n in shape]
    d2 = wide.L(dt) ** 2
    for _ in range(steps):
        up = 2 * u - um + d2 / r * wide.operator(u, m, l, one, h)[0]
        up[~np.broadcast_to(wide._interior(np.ones_like(r)) > 0, up.shape)] = 0
        new = up + d2 / 12 / r * wide.operator(up - 2 * u + um, m, l, one, h)[0]
        u, um = new, u
    error = {}
    for form in (sg.STAGES_FIXED, sg.STAGES_FP64):
        ew = sg.EW(sg.grid_desc(nx, ny, nz, h, bc=(1,) * 6, sg_gp=4))
        ew.set_stage_form(form)
        ew.set_material(*[dev(a) for a in mat])
        ew.set_time_step(dt, 0.0)
        got = _steps(ew, *fields, steps).reshape(u.shape)
        ew.close()
        e = got[cut] - u[cut]
        error[form] = float(np.sqrt(np.sum(e * e) / np.sum(u[cut] ** 2)))
    assert error[sg.STAGES_FIXED] <= error[sg.STAGES_FP64] < 1e-14, error
