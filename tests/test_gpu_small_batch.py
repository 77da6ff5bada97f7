"""Batches of small circuits too large for the cluster sweeps: a launch per pass with as many
warps as its tasks need.  Every member has the bits of the same evaluation alone (cluster sweeps),
from passes of one task up to a task per warp, half passes and full ones side by side."""
import numpy as np
import pytest

from tests.fixtures import synthetic_problem
from tests.test_gpu_half_passes import compressed_angles, make_engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,na,nb,layers,cplx", [(2, 1, 1, 1, False), (4, 2, 2, 2, True), (7, 3, 4, 1, False),
                                                 (8, 4, 4, 2, False), (8, 4, 4, 1, True), (9, 3, 3, 1, False)])
def test_members_have_the_bits_of_one(N, na, nb, layers, cplx):
    pb = synthetic_problem(N, na, nb, layers, 9)
    P = int(np.max(pb["order_1b"]))
    rng = np.random.default_rng(N + nb)
    rows = 11
    ang = np.stack([compressed_angles(pb, rng.uniform(-1.0, 1.0, P)) for _ in range(rows)])
    ang[::2] += rng.uniform(-0.3, 0.3, ang[::2].shape)
    bat, one = make_engine(pb, rows, cplx), make_engine(pb, 1, cplx)
    for e in (bat, one):
        e.set_ham_integrals(pb["h1"], pb["g2"])
    E, g = bat.gradient(ang)
    for b in range(rows):
        E1, g1 = one.gradient(ang[b])
        assert E[b] == E1 and np.array_equal(g[b], g1)
    bat.close()
    one.close()
