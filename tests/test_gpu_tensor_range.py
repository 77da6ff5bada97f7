"""Single elements of H x from the tensor-core product: vectors with a tail of small elements
get the FP64 kernels' result bit for bit, through every call that returns H x; for vectors of
one scale the product's error by element, against sums in extended precision, is no larger than
the FP64 kernels'."""
import numpy as np
import pytest

import ansatzevolve_gb300 as ae
from ansatzevolve_gb300.synthetic import hartree_fock_index
from tests.fixtures import oracle_synthetic, synthetic_problem
from tests.test_gpu_streams import make

pytestmark = pytest.mark.gpu


def vectors(e, N, na, nb, rng):
    """Name, vector: all of too wide a range."""
    D, W = e.D, e.W
    hf = hartree_fock_index(N, na, nb)
    # excitations away from the reference determinant; H reaches two further at a time
    rank = np.array([bin(int(z) ^ hf).count("1") // 2 for z in e.states()])
    steps = np.repeat((rank + 1) // 2, W)
    x = rng.standard_normal(D * W)
    yield "falling by 1e-3 an application of H", x * 1e-3 ** steps
    yield "falling by 1e-4", x * 1e-4 ** steps
    yield "one determinant", np.where(np.repeat(rank == 0, W), 1.0, 0.0)
    yield "odd excitations small", x * np.where(np.repeat(rank, W) % 2, 1e-9, 1.0)
    yield "every fifth amplitude zero", x * (np.repeat(np.arange(D), W) % 4 > 0)
    yield "one dominant amplitude", np.where(np.repeat(rank == 0, W), 1.0, 1e-3 * x / np.sqrt(D))


@pytest.mark.parametrize("N,na,nb,cplx", [(8, 4, 4, False), (9, 5, 4, False), (8, 4, 3, True), (10, 5, 5, False)])
def test_wide_ranges_are_the_fp64_kernels(monkeypatch, N, na, nb, cplx):
    torch = pytest.importorskip("torch")
    e, ref = (make(monkeypatch, t, N, na, nb, cplx) for t in (True, False))
    rng = np.random.default_rng(N)
    st = torch.cuda.Stream()
    for name, v in vectors(e, N, na, nb, rng):
        for scale in (1.0, 1e-100):
            y = e.apply_h(scale * v)
            assert not e.tensor_status()[0], name
            assert np.array_equal(y, ref.apply_h(scale * v)), name
        # on the device, with the spin-flip symmetric vector's half product and <x|y>
        for sym in (False, True):
            if sym and na != nb:
                continue
            u = v.reshape(-1, e.W)
            if sym:
                n = int(round(np.sqrt(e.D)))
                u = u.reshape(n, n, e.W)
                u = (u + u.transpose(1, 0, 2)).reshape(-1, e.W)
            x = torch.from_numpy(np.ascontiguousarray(u.reshape(-1))).cuda()
            out = []
            for eng in (e, ref):
                y = torch.empty_like(x)
                E = torch.empty(1, dtype=torch.float64, device="cuda")
                torch.cuda.synchronize()
                eng.apply_dev(x.data_ptr(), y.data_ptr(), E.data_ptr(), st.cuda_stream)
                torch.cuda.synchronize()
                out.append((y.cpu().numpy(), E.item()))
            assert not e.tensor_status()[0], name
            assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1], name
    # a batch: by instance
    if not cplx:
        xs = np.stack([rng.standard_normal(e.D), next(vectors(e, N, na, nb, rng))[1], rng.uniform(-1, 1, e.D)])
        alone = [e.apply_h(v) for v in xs]
        e.set_batch(3)
        ys = np.asarray(e.apply_h(xs.reshape(-1))).reshape(3, -1)
        assert list(e.tensor_status()) == [True, False, True]
        for y, z in zip(ys, alone):
            assert np.array_equal(y, z)
    e.close()
    ref.close()


def test_knob_and_status(monkeypatch):
    e, ref = (make(monkeypatch, t, 8, 4, 4) for t in (True, False))
    x = np.random.default_rng(0).standard_normal(e.D)
    ang = np.random.default_rng(1).uniform(-0.3, 0.3, e.nops)
    assert e.get_tuning(ae.TUNE_TENSOR) == 1
    y, g = e.apply_h(x), e.gradient(ang)
    assert e.tensor_status()[0]
    e.set_tuning(ae.TUNE_TENSOR, 0)
    assert np.array_equal(e.apply_h(x), ref.apply_h(x)) and not e.tensor_status()[0]
    g0, r0 = e.gradient(ang), ref.gradient(ang)
    assert g0[0] == r0[0] and np.array_equal(g0[1], r0[1]) and not e.tensor_status()[0]
    e.set_tuning(ae.TUNE_TENSOR, 1)
    assert np.array_equal(e.apply_h(x), y)
    g1 = e.gradient(ang)
    assert g1[0] == g[0] and np.array_equal(g1[1], g[1]) and e.tensor_status()[0]
    with pytest.raises(ae.AegpuError):
        e.set_tuning(ae.TUNE_TENSOR, 2)
    e.close()
    ref.close()


def test_error_by_element(monkeypatch):
    N, na, nb = 10, 5, 4
    e, ref = (make(monkeypatch, t, N, na, nb) for t in (True, False))
    pb = synthetic_problem(N, na, nb, 1, 5)
    rowp, col, val = oracle_synthetic(pb, csr=True).csr()
    rng = np.random.default_rng(4)
    for x in (rng.standard_normal(e.D), rng.uniform(-1.0, 1.0, e.D)):
        x /= np.linalg.norm(x)
        got, fp64 = e.apply_h(x), ref.apply_h(x)
        assert e.tensor_status()[0]
        err = []
        for r0 in range(0, e.D, 2000):
            r1 = min(e.D, r0 + 2000)
            s = slice(rowp[r0], rowp[r1])
            terms = val[s].astype(np.longdouble) * x[col[s]]
            at = rowp[r0:r1] - rowp[r0]
            y = np.add.reduceat(terms, at)
            w = np.add.reduceat(np.abs(val[s] * x[col[s]]), at)
            err.append(np.stack([np.abs(got[r0:r1] - y) / w, np.abs(fp64[r0:r1] - y) / w]).astype(float))
        t, f = np.concatenate(err, axis=1)
        print("by element: tensor rms %.2e max %.2e, FP64 rms %.2e max %.2e" % (np.sqrt(np.mean(t ** 2)), t.max(),
                                                                            np.sqrt(np.mean(f ** 2)), f.max()))
        assert np.mean(t ** 2) <= np.mean(f ** 2) and t.max() <= f.max()
    e.close()
    ref.close()
