"""A problem that is refused while its passes are built leaves nothing behind: the next problem on
the same handle gives the bits of a fresh engine."""
import ctypes

import numpy as np
import pytest

import ansatzevolve_gb300 as ae
from ansatzevolve_gb300.synthetic import hartree_fock_index, synthetic_integrals, tups_operators

pytestmark = pytest.mark.gpu
N, NA, NB = 6, 3, 2


def number(p):
    return [p, p, -1, -1]


def single(p, q):
    return [p, q, -1, -1]


# number operators in two runs with rotations between, then a spin flip, which leaves the sector
REFUSED = ([number(p) for p in range(2 * N)] + [single(0, 1), single(N, N + 1)] +
           [[0, N, 0, N], [1, N + 2, 1, N + 2]] + [single(0, N)])


def engine(ops, cplx, refused):
    e = object.__new__(ae.Engine)
    e.L, e.h, e.nb = ae.lib(), ctypes.c_void_p(), 1
    assert e.L.aegpu_create(ctypes.byref(e.h)) == 0
    for o, c, expect in ([(REFUSED, 1, 5)] if refused else []) + [(ops, int(cplx), 0)]:
        o = np.ascontiguousarray(o, dtype=np.int32)
        rc = e.L.aegpu_set_problem(e.h, 2 * N, ae.BASIS_SZ, NA + NB, NA, NB, c, len(o), ae.iptr(o.reshape(-1)))
        assert rc == expect, e.L.aegpu_last_error(e.h)
    e.nops, e.W, e.D = len(o), 2 if cplx else 1, int(e.L.aegpu_dim(e.h))
    s = np.zeros(e.D * e.W)
    s[e.W * int(np.searchsorted(e.states(), hartree_fock_index(N, NA, NB)))] = 1.0
    e.set_initial(s)
    e.set_ham_integrals(*synthetic_integrals(N, 3))
    return e


@pytest.mark.parametrize("ops,cplx", [
    ([single(0, 1), single(N, N + 1), number(0), number(N + 1), single(1, 2), single(N + 1, N + 2)], True),
    ([single(0, 1), single(1, 2)], True),
    ((tups_operators(N, 1)[0] - 1).tolist(), False)])
def test_after_a_refused_problem(ops, cplx):
    one, again = (engine(ops, cplx, refused) for refused in (False, True))
    rng = np.random.default_rng(1)
    for _ in range(3):
        x = rng.uniform(-0.5, 0.5, len(ops))
        (E, g), (E1, g1) = again.gradient(x), one.gradient(x)
        assert E == E1 and np.array_equal(g, g1)
        assert np.array_equal(again.evolve(x), one.evolve(x))
    one.close()
    again.close()
