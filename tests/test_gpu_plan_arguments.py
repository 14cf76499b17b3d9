"""Every required array of a plan's description is refused when it is missing, before anything reads it."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

REQUIRED = ("Dr", "D2_r2", "ir4_r2", "D2_sine", "ir2_sine", "D2_A4", "ir2_A4", "ir4_A4", "rsq", "dT0", "gr",
            "Linv_A4", "Linv_T", "Linv_S")


@pytest.mark.parametrize("missing", REQUIRED + (None,))
def test_missing_arrays_are_refused(cuda, missing):
    import numpy as np
    from spectraldoublediffusiveconvection_gb300 import _lib
    from spectraldoublediffusiveconvection_gb300.operators import plan_arrays
    cuda.zeros(1, device="cuda")
    A = {k: np.ascontiguousarray(v) for k, v in plan_arrays(8, 6, 2.0, 1e-3, 1.0, 0.01).items()}
    L = _lib.lib()
    for precision in (_lib.SDD_PREC_FP64, _lib.SDD_PREC_MIXED):
        d = _lib.PlanDesc()
        d.N_fm, d.nr, d.precision, d.dt, d.Pr, d.Tau = 8, 5, precision, 1e-3, 1.0, 0.01
        for name in REQUIRED:
            if name != missing:
                setattr(d, name, A[name].ctypes.data_as(ctypes.POINTER(ctypes.c_double)))
        h = ctypes.c_void_p()
        st = L.sdd_plan_create(ctypes.byref(d), ctypes.byref(h))
        assert st == (_lib.SDD_OK if missing is None else _lib.SDD_ERR_ARG)
        assert (h.value is None) == (missing is not None)
        if h.value:
            assert L.sdd_plan_destroy(h) == _lib.SDD_OK
