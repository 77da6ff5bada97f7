"""A knob set to its default value changes nothing: the CTAs per SM of the pass kernels decide the
order of the gradients' sums, so the same launch shapes show as the same bits."""
import numpy as np
import pytest

import ansatzevolve_gb300 as ae
from ansatzevolve_gb300 import autotune
from ansatzevolve_gb300.synthetic import hartree_fock_index, synthetic_integrals, tups_operators

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,na,nb", [(10, 5, 5), (12, 6, 6)])
def test_default_values(N, na, nb):
    ops = tups_operators(N, 1)[0] - 1
    ang = np.random.default_rng(N).uniform(-0.5, 0.5, len(ops))
    got = []
    for tuning in (None, autotune.DEFAULT, {ae.TUNE_CTAS_PER_SM: 8}):
        e = ae.Engine(2 * N, ae.BASIS_SZ, na + nb, na, nb, ops, tuning=tuning)
        s = np.zeros(e.D)
        s[int(np.searchsorted(e.states(), hartree_fock_index(N, na, nb)))] = 1.0
        e.set_initial(s)
        e.set_ham_integrals(*synthetic_integrals(N, 5))
        got.append(e.gradient(ang))
        assert e.get_tuning(ae.TUNE_CTAS_PER_SM) == (8 if tuning and len(tuning) == 1 else 4)
        e.close()
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])
    np.testing.assert_allclose(got[0][1], got[2][1], atol=1e-11, rtol=0)
