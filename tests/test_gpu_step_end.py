"""The end of a step (dt, t, stop test) beside the last cell kernel, in the last block of a fused pass or after a
profiled step gives the same dt, t and fields: step counts of both parities, one call against many, and a run that
stops inside a captured sequence."""
import os

import numpy as np
import pytest

from ecogen_b200 import api, cases

pytestmark = pytest.mark.gpu

SPECS = {
    "tube": lambda: cases.shock_tube_1d(ncells=300, iterations=7, total_time=None),
    "tube_muscl": lambda: cases.shock_tube_1d(ncells=130, iterations=7, total_time=None, order="vanleer"),
    "bubble": lambda: cases.shock_bubble_2d(n=20, iterations=7),
    "euler": lambda: cases.euler_blast_2d(n=18, iterations=7),
    "euler_tube": lambda: cases.euler_shock_tube(ncells=140, iterations=7, order="vanleer"),
    "ptueq": lambda: cases.ptueq_bubble_2d(n=18, iterations=7),
    "ptueq_tube": lambda: cases.ptueq_shock_tube_1d(ncells=140, iterations=7),
}


@pytest.mark.parametrize("key", list(SPECS))
def test_step_end_forms_agree(key, tmp_path):
    spec = SPECS[key]()
    inp = api.Input(spec.write(str(tmp_path)), os.path.join(str(tmp_path), "libEOS"))

    def go(advance):
        ctx = api.Context(inp.case)
        ctx.upload(inp.fill())
        advance(ctx)
        out = ctx.download(), ctx.dt.value, ctx.t.value, ctx.iteration
        ctx.close()
        return out

    ref = go(lambda c: [c.step(1) for _ in range(7)])
    forms = [lambda c: c.step(7), lambda c: [c.step(3), c.step(4)], lambda c: c.step_profiled(7), lambda c: c.run()]
    for advance in forms:
        got = go(advance)
        assert got[1:] == ref[1:]
        for a, b in zip(got[0], ref[0]):
            assert np.array_equal(a, b)
