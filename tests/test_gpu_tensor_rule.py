"""Which sectors and calls run H products on the tensor cores, on both sides of the rule: few
beta strings and little work stay with the FP64 kernels' bits; several vectors of one call count
together."""
import numpy as np
import pytest

import ansatzevolve_gb300 as ae
from ansatzevolve_gb300.synthetic import hartree_fock_index, synthetic_integrals, tups_operators

pytestmark = pytest.mark.gpu


def make(monkeypatch, tensor, N, na, nb, rows, cplx):
    if tensor:
        monkeypatch.delenv("AEGPU_TENSOR", raising=False)
    else:
        monkeypatch.setenv("AEGPU_TENSOR", "0")
    e = ae.Engine(2 * N, ae.BASIS_SZ, na + nb, na, nb, tups_operators(N, 1)[0] - 1, complex_mode=cplx)
    s = np.zeros(e.D * e.W)
    s[e.W * int(np.searchsorted(e.states(), hartree_fock_index(N, na, nb)))] = 1.0
    e.set_initial(s)
    if rows > 1:
        e.set_batch(rows)
    e.set_ham_integrals(*synthetic_integrals(N, 5))
    return e


@pytest.mark.parametrize("N,na,nb,rows,cplx,tensor", [
    (12, 6, 1, 1, False, False), (12, 6, 1, 32, False, False), (13, 3, 12, 1, True, False), (13, 3, 2, 1, False, False),
    (13, 3, 2, 2, False, True), (13, 3, 2, 1, True, True), (10, 4, 3, 1, False, True), (10, 5, 2, 1, False, False), (10, 5, 2, 12, False, True),
    (10, 5, 3, 1, False, True), (10, 5, 5, 1, False, True), (9, 5, 5, 16, False, False)])
def test_rule(monkeypatch, N, na, nb, rows, cplx, tensor):
    e, ref = (make(monkeypatch, t, N, na, nb, rows, cplx) for t in (True, False))
    rng = np.random.default_rng(N)
    x = rng.standard_normal(rows * e.D * e.W)
    ang = rng.uniform(-0.3, 0.3, (rows, e.nops))
    y, z = e.apply_h(x), ref.apply_h(x)
    assert list(e.tensor_status()) == [tensor] * rows
    (E, g), (Er, gr) = e.gradient(ang), ref.gradient(ang)
    assert list(e.tensor_status()) == [tensor] * rows
    if tensor:
        # as in test_gpu_tensor: row widths below 2605
        assert np.linalg.norm(y - z) <= 1e-14 * np.linalg.norm(z)
        np.testing.assert_allclose(E, Er, rtol=1e-12)
        np.testing.assert_allclose(g, gr, atol=1e-12, rtol=0)
    else:
        assert np.array_equal(y, z) and np.array_equal(E, Er) and np.array_equal(g, gr)
    e.close()
    ref.close()
