"""New integrals on an engine: which product they get depends on them alone, not on what the
engine held before.  Sequences of integrals that the tensor-core product takes (A, B) and
refuses (without the symmetry; with a value that is not finite; above 1e100, found when its
tables are built) give the bits, and hold the memory, of an engine that was given only them."""
import numpy as np
import pytest

import ansatzevolve_gb300 as ae
from ansatzevolve_gb300.synthetic import hartree_fock_index, synthetic_integrals, tups_operators

pytestmark = pytest.mark.gpu
N, NA, NB = 8, 4, 4


def integrals(kind):
    h1, g2 = synthetic_integrals(N, 1 if kind == "A" else 2)
    g2 = g2.copy()
    if kind == "asymmetric":
        g2[0, 1, 2, 3] += 1e-3
    elif kind == "infinite":
        g2[0, 0, 1, 1] = np.inf
    elif kind == "huge":
        g2 *= 1e101
    return h1, g2


def make(nb=1, cplx=False):
    e = ae.Engine(2 * N, ae.BASIS_SZ, NA + NB, NA, NB, tups_operators(N, 1)[0] - 1, complex_mode=cplx)
    s = np.zeros(e.D * e.W)
    s[e.W * int(np.searchsorted(e.states(), hartree_fock_index(N, NA, NB)))] = 1.0
    e.set_initial(s)
    if nb > 1:
        e.set_batch(nb)
    return e


@pytest.mark.parametrize("mode", [ae.HAM_STORED, ae.HAM_ON_THE_FLY])
@pytest.mark.parametrize("refused", ["asymmetric", "infinite", "huge"])
def test_refused_and_accepted_in_turn(monkeypatch, mode, refused):
    monkeypatch.setenv("AEGPU_TENSOR", "1")
    rng = np.random.default_rng(7)
    ang = rng.uniform(-0.3, 0.3, len(tups_operators(N, 1)[0]))
    e = make()
    for kind in ("A", refused, "A", "B", refused, refused, "B"):
        h1, g2 = integrals(kind)
        e.set_ham_integrals(h1, g2, mode)
        one = make()
        one.set_ham_integrals(h1, g2, mode)
        for x in (ang, 0.5 * ang):
            E, g = e.gradient(x)
            E1, g1 = one.gradient(x)
            assert np.array_equal(E, E1, equal_nan=True) and np.array_equal(g, g1, equal_nan=True), kind
        assert e.tensor_status()[0] == one.tensor_status()[0]
        if kind != "infinite":
            assert e.tensor_status()[0] == (kind != refused)
        assert e.device_bytes() == one.device_bytes(), kind
        one.close()
    e.close()


def test_refused_member_of_a_batch(monkeypatch):
    monkeypatch.setenv("AEGPU_TENSOR", "1")
    ang = np.random.default_rng(8).uniform(-0.3, 0.3, (3, len(tups_operators(N, 1)[0])))
    sets = [["A", "B", "A"], ["A", "asymmetric", "B"], ["B", "A", "A"]]
    e = make(3)
    for kinds in sets:
        h, g = zip(*(integrals(k) for k in kinds))
        e.set_ham_integrals_batch(np.stack(h), np.stack(g))
        one = make(3)
        one.set_ham_integrals_batch(np.stack(h), np.stack(g))
        (E, d), (E1, d1) = e.gradient(ang), one.gradient(ang)
        assert np.array_equal(E, E1) and np.array_equal(d, d1)
        assert list(e.tensor_status()) == ["asymmetric" not in kinds] * 3
        one.close()
    e.close()
