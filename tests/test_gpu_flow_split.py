"""The Euler and PTUEq models in split form (per-axis face kernels and a cell kernel) against their fused
kernels, bit for bit, at the sizes where the face tiles end, staged by tensor copies (even x) and by plain
loads, with symmetry sides, every limiter and first order.

The fused kernels run the same case when it carries a passive transport (Euler), or when its limiter slots
differ in name only: THINC as the interface limiter of p, T and u limits as minmod does (PTUEq)."""
import os

import numpy as np
import pytest

from ecogen_b200 import api, cases

pytestmark = pytest.mark.gpu

CELLS = [(3, 2, 1), (15, 9, 1), (16, 8, 1), (17, 33, 1), (32, 16, 1), (4, 17, 9), (18, 7, 24)]


def _run(spec, fields):
    rec = api.case_from_spec(spec)
    ctx = api.Context(rec)
    ctx.upload(fields)
    st = ctx.step(6)
    out = ctx.download_dict()
    res = out, ctx.dt.value, st.nonfinite_cells
    ctx.close()
    return res


def _fill(spec, tmp):
    inp = api.Input(spec.write(str(tmp)), os.path.join(str(tmp), "libEOS"))
    return inp.fill()


def _same(a, b):
    assert a[1] == b[1] and a[2] == b[2] == 0
    for name in ("alpha", "rho", "p", "u", "E"):
        assert np.array_equal(a[0][name], b[0][name]), name


@pytest.mark.parametrize("order", [None, "vanleer", "superbee", "vanalbada", "mc"])
@pytest.mark.parametrize("cells", CELLS)
def test_euler_split_equals_fused(cells, order, tmp_path):
    spec = cases.euler_blast_2d(n=cells[0], ny=cells[1], nz=cells[2], iterations=6, order=order)
    spec.boundaries = ["wall", "nonReflecting", "symmetry", "wall", "nonReflecting", "symmetry"]
    f = _fill(spec, tmp_path)
    split = _run(spec, f)
    spec.transports = ["t"]
    _same(split, _run(spec, f + [np.linspace(0.0, 1.0, len(f[0]))]))


@pytest.mark.parametrize("cells", CELLS)
def test_ptueq_split_equals_fused(cells, tmp_path):
    spec = cases.ptueq_bubble_2d(n=cells[0], ny=cells[1], nz=cells[2], iterations=6, limiter="minmod")
    f = _fill(spec, tmp_path)
    split = _run(spec, f)
    spec.interface_limiter, spec.vf_limiter, spec.interface_vf_limiter = "THINC", "minmod", "minmod"
    _same(split, _run(spec, f))
