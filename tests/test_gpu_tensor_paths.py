"""The schedules of the tensor-core product that follow the vector: spin-flip symmetric vectors
(half of the alpha-beta part, the alpha part as a transpose) in sectors whose rows are summed in
shared memory and, above 1024 strings, in global memory; batches whose members take different
schedules; and a vector whose digit sums leave the window of the integer read-out, so that the
FP64 kernels follow the product.

Tolerance of the comparisons with the FP64 kernels: as in test_gpu_tensor.py, 1e-14 of |y| in
the 2-norm for rows of up to 2605 elements (13 orbitals: 2479)."""
import itertools

import numpy as np
import pytest

import ansatzevolve_gb300 as ae
from ansatzevolve_gb300.synthetic import hartree_fock_index, synthetic_integrals, tups_operators
from tests.fixtures import synthetic_problem
from tests.test_gpu_half_passes import compressed_angles

pytestmark = pytest.mark.gpu
TOL = 1e-14


def make(monkeypatch, tensor, N, n, cplx=False, mode=ae.HAM_AUTO, integrals=None, rows=1):
    monkeypatch.setenv("AEGPU_TENSOR", "1" if tensor else "0")
    e = ae.Engine(2 * N, ae.BASIS_SZ, 2 * n, n, n, tups_operators(N, 1)[0] - 1, complex_mode=cplx)
    s = np.zeros(e.D * e.W)
    s[e.W * int(np.searchsorted(e.states(), hartree_fock_index(N, n, n)))] = 1.0
    e.set_initial(s)
    if rows > 1:
        e.set_batch(rows)
    e.set_ham_integrals(*(integrals or synthetic_integrals(N, 5)), mode)
    return e


@pytest.mark.parametrize("N,n,cplx,mode", [(8, 4, False, ae.HAM_AUTO), (8, 4, True, ae.HAM_ON_THE_FLY),
                                           (9, 6, False, ae.HAM_AUTO), (10, 5, True, ae.HAM_AUTO),
                                           (13, 6, False, ae.HAM_ON_THE_FLY)])
def test_symmetric_vectors(monkeypatch, N, n, cplx, mode):
    torch = pytest.importorskip("torch")
    got, want = (make(monkeypatch, t, N, n, cplx, mode) for t in (True, False))
    ns = int(round(np.sqrt(got.D)))
    u = np.random.default_rng(N).standard_normal((ns, ns, got.W))
    sym = u + u.transpose(1, 0, 2)
    near = sym.copy()
    near[0, 1] += 1e-6  # outside the test's 1e-12
    for v in (sym, near, u):
        x = torch.from_numpy(np.ascontiguousarray(v.reshape(-1))).cuda()
        out = []
        for e in (got, want):
            y, E = torch.empty_like(x), torch.empty(1, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            e.apply_dev(x.data_ptr(), y.data_ptr(), E.data_ptr(), torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            out.append((y, E))
        assert got.tensor_status()[0]
        (y, E), (z, F) = out
        assert torch.linalg.norm(y - z) <= TOL * torch.linalg.norm(z)
        assert abs(E - F) <= TOL * torch.linalg.norm(z) * torch.linalg.norm(x)
    got.close()
    want.close()


def test_batch_of_different_schedules(monkeypatch):
    """Symmetric and other members, one with NaN angles and one masked, in every order of a first
    three: each member has the bits of the same evaluation alone."""
    pb = synthetic_problem(8, 4, 4, 1, 5)
    rng = np.random.default_rng(2)
    P = int(np.max(pb["order_1b"]))
    sym = [compressed_angles(pb, rng.uniform(-0.5, 0.5, P)) for _ in range(2)]
    other = [s + rng.uniform(-0.3, 0.3, len(s)) for s in sym]
    nan = sym[0].copy()
    nan[3] = np.nan
    bat, one = make(monkeypatch, True, 8, 4, rows=6), make(monkeypatch, True, 8, 4)
    alone = {id(a): one.gradient(a) for a in sym + other}
    for first in itertools.permutations([sym[0], other[0], nan]):
        rows = list(first) + [sym[1], other[1], sym[0]]
        bat.set_active([1, 1, 1, 1, 1, 0])
        E, g = bat.gradient(np.stack(rows))
        for b, a in enumerate(rows[:5]):
            if a is nan:
                assert np.isnan(E[b])
                continue
            assert E[b] == alone[id(a)][0] and np.array_equal(g[b], alone[id(a)][1])
        assert [bool(u) for u in bat.tensor_status()[:5]] == [a is not nan for a in rows[:5]]
        assert [bool(u) for u in bat.flip_status()[:5]] == [any(a is s for s in sym) for a in rows[:5]]
    bat.close()
    one.close()


def test_sums_outside_the_window(monkeypatch):
    """Integrals and amplitudes whose base-512 digits are 255 throughout, the amplitudes' signs
    those of the 20 rows that one beta string meets: the five digit products of group 4 add up to
    20 (4 * 255^2 + 255) = 5.2e6 units, above the window of 2^22."""
    N, n = 8, 4
    digits = lambda k, lead: lead / 512 + sum(255.0 / 512.0 ** (i + 1) for i in range(1, k))
    g2 = np.full((N,) * 4, 255.0 / 512 + digits(6, 0))  # scale 1
    ints = (np.zeros((N, N)), g2)
    got, want = (make(monkeypatch, t, N, n, integrals=ints) for t in (True, False))
    strings = sorted(sum(1 << i for i in c) for c in itertools.combinations(range(N), n))
    rank = {s: i for i, s in enumerate(strings)}
    b0 = strings[17]
    c = 256 * digits(6, 1)  # the norm factor 3.3 of 70 amplitudes of 0.75 gives a scale of 256
    x = np.full((len(strings), len(strings)), c)
    for p in range(N):
        for r in range(N):
            if (b0 >> p) & 1 and not (b0 >> r) & 1:
                lo, hi = min(p, r), max(p, r)
                between = ((1 << hi) - 1) & ~((2 << lo) - 1)
                if bin(b0 & between).count("1") & 1:
                    x[:, rank[b0 ^ (1 << p) ^ (1 << r)]] = -c
    y, z = got.apply_h(x.reshape(-1)), want.apply_h(x.reshape(-1))
    assert not got.tensor_status()[0]
    assert np.array_equal(y, z)
    # digits without a pattern stay in the window
    v = np.random.default_rng(3).standard_normal(x.size)
    y, z = got.apply_h(v), want.apply_h(v)
    assert got.tensor_status()[0]
    assert np.linalg.norm(y - z) <= TOL * np.linalg.norm(z)
    got.close()
    want.close()
