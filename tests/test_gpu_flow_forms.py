"""The form and staging of Euler and PTUEq steps on 2D and 3D meshes as the C ABI reports, sets and times them:
split is what runs by default and what ecg_step_form answers, fused runs when it is asked for, and both, and both
stagings of the split form, give the same bits."""
import os

import numpy as np
import pytest

from ecogen_b200 import api, cases

pytestmark = pytest.mark.gpu

CELLS = [(2, 2, 1), (17, 33, 1), (32, 16, 1), (18, 7, 24)]
SIDES = ["symmetry", "nonReflecting", "wall", "symmetry", "nonReflecting", "symmetry"]


def _euler(cells, limiter):
    c = cases.euler_blast_2d(n=cells[0], ny=cells[1], nz=cells[2], iterations=6, order=limiter)
    c.boundaries = SIDES[:2 * c.dim]
    return c


def _ptueq(cells, limiter):
    c = cases.ptueq_bubble_2d(n=cells[0], ny=cells[1], nz=cells[2], iterations=6, limiter=limiter)
    if limiter is None:  # MUSCL runs without symmetry sides
        c.boundaries = SIDES[:2 * c.dim]
    return c


def _context(spec, tmp):
    inp = api.Input(spec.write(str(tmp)), os.path.join(str(tmp), "libEOS"))
    return api.Context(inp.case), inp.fill()


def _six(ctx, f):
    ctx.upload(f)
    ctx.dt.value, ctx.t.value = 1e-15, 0.0
    assert ctx.step(6).nonfinite_cells == 0
    return ctx.download(), ctx.dt.value, ctx.t.value


def _same(a, b):
    assert a[1:] == b[1:]
    for x, y in zip(a[0], b[0]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("limiter", [None, "vanleer", "minmod", "superbee"])
@pytest.mark.parametrize("cells", CELLS)
@pytest.mark.parametrize("make", [_euler, _ptueq])
def test_forms_and_stagings_give_the_same_bits(make, cells, limiter, tmp_path):
    ctx, f = _context(make(cells, limiter), tmp_path)
    staged = api.STAGING_TMA if cells[0] % 2 == 0 else api.STAGING_PLAIN
    assert ctx.step_form == api.FORM_SPLIT and ctx.face_staging == staged
    ref = _six(ctx, f)
    ctx.set_face_staging(api.STAGING_PLAIN)
    assert ctx.step_form == api.FORM_SPLIT and ctx.face_staging == api.STAGING_PLAIN
    _same(ref, _six(ctx, f))
    ctx.set_face_staging(api.STAGING_TMA)
    ctx.set_step_form(api.FORM_FUSED)
    assert ctx.step_form == api.FORM_FUSED and ctx.face_staging == api.STAGING_PLAIN
    _same(ref, _six(ctx, f))
    _, ms = ctx.step_profiled_kernels(1)  # a fused pass is one kernel, in its cell slot
    assert all(v == 0.0 for i, v in enumerate(ms) if i not in (3, 7, 8)) and ms[3] > 0.0
    ctx.set_step_form(api.FORM_SPLIT)
    assert ctx.step_form == api.FORM_SPLIT and ctx.face_staging == staged
    _same(ref, _six(ctx, f))
    _, ms = ctx.step_profiled_kernels(1)
    dim, two = 2 + (cells[2] > 1), limiter is not None
    run = [a for p in range(1 + two) for a in (*(4 * p + d for d in range(dim)), 4 * p + 3)] + [8]
    assert [i for i, v in enumerate(ms) if v > 0.0] == run
    ctx.close()


@pytest.mark.parametrize("transports", [False, True])
def test_cases_that_run_fused_only_say_so(transports, tmp_path):
    if transports:
        spec = _euler((16, 12, 1), "vanleer")
        spec.transports = ["t"]
    else:  # limiter slots that differ
        spec = _ptueq((16, 12, 1), "vanleer")
        spec.vf_limiter = "minmod"
    ctx, _ = _context(spec, tmp_path)
    assert ctx.step_form == api.FORM_FUSED and ctx.face_staging == api.STAGING_PLAIN
    with pytest.raises(api.EcgError):
        ctx.set_step_form(api.FORM_SPLIT)
    ctx.close()


def test_kernels_are_configured_whatever_the_order_of_settings(tmp_path):
    """A context configures the kernels of its present form and seed: every combination of the two, reached in either
    order, steps and gives the plain split form's bits where no seed is installed."""
    from ecogen_b200 import seed as seedmod
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    model = seedmod.SeedModel.load(os.path.join(root, "ecogen_b200", "models", "seed_np3.npz"))
    spec = cases.cavity_collapse_3d(n=14, iterations=6, ninclusions=3, radius_cells=(2.0, 4.0))
    ctx, f = _context(spec, tmp_path)
    ref = _six(ctx, f)
    model.install(ctx)
    ctx.set_step_form(api.FORM_FUSED)
    seeded = _six(ctx, f)
    ctx.set_seed_model(None)
    _same(ref, _six(ctx, f))
    model.install(ctx)
    ctx.set_step_form(api.FORM_SPLIT)
    _same(seeded, _six(ctx, f))
    ctx.set_seed_model(None)
    ctx.set_step_form(api.FORM_FUSED)
    _same(ref, _six(ctx, f))
    ctx.close()
