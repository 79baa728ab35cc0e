"""Batched cases at the edges of the batch kernels' blocks: cell counts around multiples of tile - 1 faces and
of 128 cells, for every tile, against the same case advanced alone (fused kernels), bit for bit."""
import ctypes as C

import numpy as np
import pytest

from ecogen_b200 import api, cases

pytestmark = pytest.mark.gpu

SIZES = (2, 3, 61, 62, 63, 64, 126, 127, 128, 129, 254, 255, 256, 381)


def _fields(spec, tmp, name):
    import os
    inp = api.Input(spec.write(str(tmp), subdir=name), os.path.join(str(tmp), "libEOS"))
    return inp.case, inp.fill()


@pytest.mark.parametrize("order", [None, "vanleer", "minmod"])
@pytest.mark.parametrize("tile", [64, 128, 256])
def test_batch_tile_edges_equal_single_runs(tile, order, tmp_path):
    specs = [cases.shock_tube_1d(ncells=n, iterations=6, order=order, x_interface=0.45) for n in SIZES]
    recs, fields = zip(*[_fields(s, tmp_path, f"c{i}") for i, s in enumerate(specs)])
    L, dp = api.lib(), C.POINTER(C.c_double)
    h = C.c_void_p()
    api.check(L.ecg_batch_create((api.Case * len(recs))(*recs), len(recs), C.byref(h)), "create")
    api.check(L.ecg_batch_set_shape(h, tile, 0), "shape")
    cat = [np.concatenate([f[k] for f in fields]) for k in range(len(fields[0]))]
    total = len(cat[0])
    api.check(L.ecg_batch_upload_prim(h, api._field_ptrs(cat), total), "upload")
    dt, t = np.full(len(recs), 1e-15), np.zeros(len(recs))
    api.check(L.ecg_batch_step(h, 6, dt.ctypes.data_as(dp), t.ctypes.data_as(dp), None), "step")
    out = [np.zeros(total) for _ in cat]
    api.check(L.ecg_batch_download_prim(h, api._field_ptrs(out), total), "download")
    L.ecg_batch_destroy(h)
    off = 0
    for i, (rec, f) in enumerate(zip(recs, fields)):
        ctx = api.Context(rec)
        ctx.upload(f)
        ctx.step(6)
        alone = ctx.download()
        n = SIZES[i]
        assert ctx.dt.value == dt[i] and ctx.t.value == t[i], n
        for k, g in enumerate(alone):
            assert np.array_equal(g, out[k][off:off + n]), (n, k)
        ctx.close()
        off += n
