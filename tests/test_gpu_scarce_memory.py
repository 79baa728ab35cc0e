"""Cases whose state fits the GPU's free memory but whose face arrays do not: the context runs the fused kernels,
with the same bits as with memory to spare."""
import os

import numpy as np
import pytest
import torch

from ecogen_b200 import api, cases

pytestmark = pytest.mark.gpu


class Scarce:
    """Leaves `left` bytes of the GPU's memory free."""

    def __init__(self, left):
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        self.held = torch.empty(max(free - left, 0), dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *a):
        self.held = None
        torch.cuda.empty_cache()


def _steps(ctx, f):
    ctx.upload(f)
    assert ctx.step(3).nonfinite_cells == 0
    return ctx.download(), ctx.dt.value


@pytest.mark.parametrize("model", ["euler", "ptueq", "kapila"])
def test_context_without_room_for_face_arrays_runs_fused(model, tmp_path):
    n = (128, 120, 126)
    if model == "euler":
        spec, planes, faces = cases.euler_blast_2d(n=n[0], ny=n[1], nz=n[2], iterations=3), 3 * 6 + 1, 15
    elif model == "ptueq":
        spec, planes, faces = cases.ptueq_bubble_2d(n=n[0], ny=n[1], nz=n[2], iterations=3), 3 * 8 + 2, 18
    else:
        spec, planes, faces = cases.shock_bubble_2d(n=1400, iterations=3), 3 * 8 + 1, 22
        n = spec.cells
    inp = api.Input(spec.write(str(tmp_path)), os.path.join(str(tmp_path), "libEOS"))
    f = inp.fill()
    ctx = api.Context(inp.case)
    assert ctx.step_form == api.FORM_SPLIT
    ref = _steps(ctx, f)
    ctx.set_step_form(api.FORM_FUSED)  # its kernels' code is on the GPU from here on
    ctx.step(1)
    ctx.close()
    cells = n[0] * n[1] * n[2]
    room = 0.6 * faces * 8 * cells  # some of the face arrays would fit
    with Scarce(int(planes * 8 * cells + room)):
        ctx = api.Context(inp.case)
        assert ctx.step_form == api.FORM_FUSED
        got = _steps(ctx, f)
        with pytest.raises(api.EcgError):
            ctx.set_step_form(api.FORM_SPLIT)
        ctx.close()
    assert got[1] == ref[1]
    for x, y in zip(got[0], ref[0]):
        assert np.array_equal(x, y)
