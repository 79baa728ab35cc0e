"""Limited slopes per cell (split form, one limiter compiled in) against the fused form's per-face ones, bit
for bit, at the sizes where the face tiles end (chunks of 16 X faces and 8 lines, 8 Y faces and 16 lines),
with symmetry sides, and with a liquid in tension, whose pressure lies below the gas phase's floor so that
the phase pressures have slopes of their own."""
import os

import numpy as np
import pytest

from ecogen_b200 import api, cases

pytestmark = pytest.mark.gpu


def _advance(spec, tmp, form, tension):
    inp = api.Input(spec.write(str(tmp)), os.path.join(str(tmp), "libEOS"))
    f = inp.fill()
    if tension:  # every third line of cells along each axis at -2e5 Pa, its energy with it
        k = np.arange(inp.ncells)
        m = ((k % spec.cells[0]) % 3 == 0) | ((k // spec.cells[0]) % 3 == 0)
        np_ = spec.nphases
        f[2 * np_ + 4][m] -= (f[2 * np_][m] + 2e5) / ((spec.eos[0].gamma - 1.0) * f[np_][m])
        f[2 * np_][m] = -2e5
    ctx = api.Context(inp.case)
    ctx.set_step_form(form)
    ctx.upload(f)
    st = ctx.step(5)
    out = (ctx.download_dict(), st.as_dict(), ctx.dt.value)
    ctx.close()
    return out


@pytest.mark.parametrize("tension", [False, True])
@pytest.mark.parametrize("cells", [(3, 2, 1), (15, 9, 1), (16, 8, 1), (17, 33, 1), (31, 16, 1), (4, 17, 9)])
def test_limited_slopes_equal_per_face_limiting(cells, tension, tmp_path):
    if cells[2] > 1:
        spec = cases.cavity_collapse_3d(n=16, iterations=5, ninclusions=4, radius_cells=(2.0, 4.0))
    else:
        spec = cases.shock_bubble_2d(n=16, iterations=5)
        spec.boundaries = ["wall", "nonReflecting", "symmetry", "wall"]
    spec.cells = cells
    (tmp_path / "a").mkdir()
    (tmp_path / "b").mkdir()
    (a, sa, da), (b, sb, db) = (_advance(spec, tmp_path / d, form, tension)
                                for d, form in (("a", api.FORM_SPLIT), ("b", api.FORM_FUSED)))
    assert sa["nonfinite_cells"] == 0 and da == db
    assert sa["newton_evals"] == sb["newton_evals"]
    for name in ("alpha", "rho", "p", "u", "E"):
        assert np.array_equal(a[name], b[name]), name
