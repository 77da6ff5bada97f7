"""Device memory that the tensor-core product holds is given back to a call that finds none left:
the call succeeds, and the engine goes on with the FP64 kernels until new integrals."""
import numpy as np
import pytest

import ansatzevolve_gb300 as ae
from ansatzevolve_gb300.synthetic import synthetic_integrals
from tests.test_gpu_streams import make

pytestmark = pytest.mark.gpu


def test_memory_is_given_back(monkeypatch):
    N = 8
    e, ref = (make(monkeypatch, t, N, 4, 4) for t in (True, False))
    ang = np.random.default_rng(1).uniform(-0.3, 0.3, e.nops)
    E, g = e.gradient(ang)
    held = e.device_bytes()
    L = ae.lib()
    try:
        L.aegpu_debug_fail_alloc_after(0)
        x = e.real_energy(ang)  # one allocation, its scratch
    finally:
        L.aegpu_debug_fail_alloc_after(-1)
    assert abs(x - E) <= 1e-12 * abs(E)
    assert e.device_bytes() < held and not e.tensor_status()[0]
    for scale in (0.5, 1.0):  # (at the same angles H psi is kept)
        (E1, g1), (E2, g2) = e.gradient(scale * ang), ref.gradient(scale * ang)
        assert E1 == E2 and np.array_equal(g1, g2)
    monkeypatch.setenv("AEGPU_TENSOR", "1")
    e.set_ham_integrals(*synthetic_integrals(N, 5))
    E1, g1 = e.gradient(ang)
    assert e.tensor_status()[0] and E1 == E and np.array_equal(g1, g)
    # without the product a failed allocation is an error, as before
    try:
        L.aegpu_debug_fail_alloc_after(0)
        with pytest.raises(ae.AegpuError):
            ref.real_energy(ang)
    finally:
        L.aegpu_debug_fail_alloc_after(-1)
    e.close()
    ref.close()
