"""Steps launched one by one, replayed from captured graphs, or both in one call give the same bits: step counts on either
side of the change-over and of both parities, in one call and in many, and after a change that drops the graphs."""
import os

import numpy as np
import pytest

from ecogen_b200 import api, cases

pytestmark = pytest.mark.gpu

N = 75  # past the first 32 steps, which run without graphs
SPECS = {
    "tube": lambda: cases.shock_tube_1d(ncells=300, iterations=50, total_time=None),
    "bubble": lambda: cases.shock_bubble_2d(n=20, iterations=50),
    "cavity": lambda: cases.cavity_collapse_3d(n=8, iterations=50, ninclusions=2),
    "euler": lambda: cases.euler_blast_2d(n=18, iterations=50),
    "ptueq": lambda: cases.ptueq_bubble_2d(n=18, iterations=50),
}


@pytest.mark.parametrize("key", list(SPECS))
def test_direct_and_captured_steps_agree(key, tmp_path):
    spec = SPECS[key]()
    inp = api.Input(spec.write(str(tmp_path)), os.path.join(str(tmp_path), "libEOS"))

    def go(advance):
        ctx = api.Context(inp.case)
        ctx.upload(inp.fill())
        advance(ctx)
        out = ctx.download(), ctx.dt.value, ctx.t.value, ctx.iteration
        ctx.close()
        return out

    def dropped(c):
        c.step(41)
        c.set_newton_cap(100)  # the default: drops the graphs
        c.step(N - 41)

    def same(got, ref):
        assert got[1:] == ref[1:]
        for a, b in zip(got[0], ref[0]):
            assert np.array_equal(a, b)

    ref = go(lambda c: c.step_profiled(N))  # never captured
    forms = [lambda c: c.step(N), lambda c: [c.step(31), c.step(1), c.step(1), c.step(42)],
             lambda c: [c.step(3) for _ in range(N // 3)], dropped]
    for advance in forms:
        same(go(advance), ref)
    same(go(lambda c: c.run()), go(lambda c: c.step_profiled(50)))  # a stop inside a captured sequence
