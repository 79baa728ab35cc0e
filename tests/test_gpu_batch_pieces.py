"""Batches whose face fluxes do not all fit the GPU's free memory run their passes in pieces, with the same bits as
with memory to spare."""
import ctypes as C
import os

import numpy as np
import pytest

from ecogen_b200 import api, cases
from tests.test_gpu_scarce_memory import Scarce

pytestmark = pytest.mark.gpu


def _batch(recs, fields):
    L, dp = api.lib(), C.POINTER(C.c_double)
    h = C.c_void_p()
    api.check(L.ecg_batch_create((api.Case * len(recs))(*recs), len(recs), C.byref(h)), "create")
    try:
        api.check(L.ecg_batch_set_shape(h, 128, 0), "shape")
        total = len(fields[0])
        api.check(L.ecg_batch_upload_prim(h, api._field_ptrs(fields), total), "upload")
        dt, t = np.full(len(recs), 1e-15), np.zeros(len(recs))
        api.check(L.ecg_batch_step(h, 5, dt.ctypes.data_as(dp), t.ctypes.data_as(dp), None), "step")
        out = [np.zeros(total) for _ in fields]
        api.check(L.ecg_batch_download_prim(h, api._field_ptrs(out), total), "download")
    finally:
        L.ecg_batch_destroy(h)
    return out, dt, t


@pytest.mark.parametrize("order", [None, "vanleer", "minmod"])
def test_batch_without_room_for_all_face_fluxes(order, tmp_path):
    """Few long tubes, so that the pieces cut through them, and short ones."""
    sizes = [2, 2_000_003, 129, 1_400_000, 128, 127, 600_001, 64]
    recs, parts = [], []
    for i, n in enumerate(sizes):
        spec = cases.shock_tube_1d(ncells=n, iterations=5, order=order, x_interface=0.45)
        inp = api.Input(spec.write(str(tmp_path), subdir=f"c{i}"), os.path.join(str(tmp_path), "libEOS"))
        recs.append(inp.case)
        parts.append(inp.fill())
    fields = [np.concatenate([p[k] for p in parts]) for k in range(len(parts[0]))]
    ref = _batch(recs, fields)
    cells = sum(sizes)
    planes = 2 * 7 + 1 + (6 if order else 0)
    with Scarce(int(planes * 8 * cells + 0.3 * 10 * 8 * cells)):
        got = _batch(recs, fields)
    assert np.array_equal(got[1], ref[1]) and np.array_equal(got[2], ref[2])
    for k, (x, y) in enumerate(zip(got[0], ref[0])):
        assert np.array_equal(x, y), k
