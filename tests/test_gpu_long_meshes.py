"""Meshes with more lines than a launch of the face kernels has blocks for (65535 along the grid's second and
third dimensions): they run fused, with the same bits as where the fused kernels run for another reason."""
import os

import numpy as np
import pytest

from ecogen_b200 import api, cases

pytestmark = pytest.mark.gpu


def _fields(rec, n):
    r = np.random.default_rng(n)
    if rec.model == api.MODEL_EULER:
        rho, p = 1. + 0.1 * r.random(n), 1e5 * (1. + 0.1 * r.random(n))
        u = [5. * r.random(n) for _ in range(3)]
        return [rho, p, *u, p / 0.4 / rho + 0.5 * sum(v * v for v in u)]
    raise ValueError(rec.model)


def _run(spec, tmp, name, extra):
    inp = api.Input(spec.write(str(tmp / name)), os.path.join(str(tmp / name), "libEOS"))
    f = _fields(inp.case, int(np.prod(spec.cells)))
    if spec.dim < 3:
        f[4][:] = 0.
        f[5] = f[1] / 0.4 / f[0] + 0.5 * (f[2] ** 2 + f[3] ** 2)
    ctx = api.Context(inp.case)
    form = ctx.step_form
    ctx.upload(f + extra(len(f[0])))
    ctx.step(2)
    out = ctx.download()[:6], ctx.dt.value
    ctx.close()
    return out, form


@pytest.mark.parametrize("cells", [(2, 8 * 65535, 1), (2, 2, 65536), (2, 65536, 2)])
def test_euler_mesh_beyond_the_face_grids(cells, tmp_path):
    spec = cases.euler_blast_2d(n=cells[0], ny=cells[1], nz=cells[2], iterations=2)
    got, form = _run(spec, tmp_path, "a", lambda n: [])
    assert form == api.FORM_FUSED
    spec.transports = ["t"]
    ref, _ = _run(spec, tmp_path, "b", lambda n: [np.linspace(0., 1., n)])
    assert got[1] == ref[1]
    for x, y in zip(got[0], ref[0]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("cells", [(2, 8 * 65535 - 1, 1), (2, 2, 65535), (2, 65535, 2)])
def test_the_longest_mesh_of_the_face_grids_runs_split(cells, tmp_path):
    spec = cases.euler_blast_2d(n=cells[0], ny=cells[1], nz=cells[2], iterations=2)
    got, form = _run(spec, tmp_path, "a", lambda n: [])
    assert form == api.FORM_SPLIT
    spec.transports = ["t"]
    ref, _ = _run(spec, tmp_path, "b", lambda n: [np.linspace(0., 1., n)])
    assert got[1] == ref[1]
    for x, y in zip(got[0], ref[0]):
        assert np.array_equal(x, y)


def test_long_ptueq_mesh_runs(tmp_path):
    spec = cases.ptueq_bubble_2d(n=2, ny=8 * 65535, nz=1, iterations=2)
    inp = api.Input(spec.write(str(tmp_path)), os.path.join(str(tmp_path), "libEOS"))
    ctx = api.Context(inp.case)
    assert ctx.step_form == api.FORM_FUSED
    ctx.upload(inp.fill())
    assert ctx.step(2).nonfinite_cells == 0
    ctx.close()
