"""The quick forms of the Newton evaluation and of the internal face against the general ones, bit for bit
(ecogen_b200/probe/ecg_quick_check.cu): ordinary states, states at and below the floors, and zero, infinite
and NaN operands, which the quick forms must leave to the general ones or solve alike."""
import ctypes as C
import os

import pytest

from ecogen_b200 import api, cases

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROBE = os.path.join(ROOT, "ecogen_b200", "libecg_probe.so")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [0.0, 1e-15])
@pytest.mark.parametrize("eos", [(cases.WATER_SG, cases.AIR_IG), (cases.LIQ_PC, cases.VAP_PC),
                                 (cases.WATER_NASG, cases.AIR_IG), (cases.WATER_SG, cases.AIR_IG, cases.GAS_B_IG)],
                         ids=lambda e: "-".join(q.kind for q in e))
def test_quick_forms_equal_general_forms(eos, eps):
    lib = C.CDLL(PROBE)
    lib.ecg_probe_quick_check.argtypes = [C.c_ulonglong, C.c_int, C.POINTER(api.Eos), C.c_double, C.c_int, C.c_int,
                                          C.POINTER(C.c_ulonglong)]
    rec = (api.Eos * len(eos))(*[api.Eos(api.EOS_CODE[e.kind], e.gamma, e.pinf, e.b, e.cv, e.eref, e.sref) for e in eos])
    counts = (C.c_ulonglong * 4)()
    assert lib.ecg_probe_quick_check(0x51 + len(eos), len(eos), rec, eps, 148 * 4, 64, counts) == 0
    states, newton, face, quick = list(counts)
    assert states == 148 * 4 * 128 * 64
    assert newton == 0, f"{newton} of {states} relaxations differ"
    assert face == 0, f"{face} of {states} faces differ"
    assert quick == 0 if any(e.kind == "NASG" for e in eos) else quick > 0.8 * states
