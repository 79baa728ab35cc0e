"""The step kernels' per-block reduction of the relaxation counters, for every block size a tile may have, against the
same counters added one by one (ecogen_b200/probe/ecg_counters_check.cu)."""
import ctypes as C
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROBE = os.path.join(ROOT, "ecogen_b200", "libecg_probe.so")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [32, 64, 128, 256, 512, 1024])
@pytest.mark.parametrize("blocks", [1, 301])
def test_block_counters_of_every_block_size(threads, blocks):
    lib = C.CDLL(PROBE)
    lib.ecg_probe_counters.argtypes = [C.c_ulonglong, C.c_int, C.c_int, C.c_ulonglong * 24, C.c_ulonglong * 24]
    got, want = (C.c_ulonglong * 24)(), (C.c_ulonglong * 24)()
    assert lib.ecg_probe_counters(0xC0 + threads, blocks, threads, got, want) == 0
    assert list(got) == list(want) and want[0] > 0
