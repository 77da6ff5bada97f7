"""H products and evaluations of one engine on several streams without any order between
them, and recorded into a caller's graph: the tensor-core product's workspace is shared, so
every result has to be the one of the same call made alone, bit for bit."""
import ctypes

import numpy as np
import pytest

import ansatzevolve_gb300 as ae
from ansatzevolve_gb300.synthetic import hartree_fock_index, synthetic_integrals, tups_operators

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def make(monkeypatch, tensor, N, na, nb, cplx=False):
    monkeypatch.setenv("AEGPU_TENSOR", "1" if tensor else "0")
    e = ae.Engine(2 * N, ae.BASIS_SZ, na + nb, na, nb, tups_operators(N, 1)[0] - 1, complex_mode=cplx)
    s = np.zeros(e.D * e.W)
    s[e.W * int(np.searchsorted(e.states(), hartree_fock_index(N, na, nb)))] = 1.0
    e.set_initial(s)
    e.set_ham_integrals(*synthetic_integrals(N, 5))
    return e


@pytest.mark.parametrize("N,na,nb,cplx", [(10, 5, 4, False), (9, 5, 4, True), (10, 5, 5, False)])
def test_unordered_streams(monkeypatch, N, na, nb, cplx):
    e = make(monkeypatch, True, N, na, nb, cplx)
    rng = np.random.default_rng(N)
    x = [torch.from_numpy(10.0 ** k * rng.standard_normal(e.D * e.W)).cuda() for k in range(4)]
    want = [torch.empty_like(v) for v in x]
    st = [torch.cuda.Stream() for _ in range(4)]
    ang = torch.from_numpy(rng.uniform(-0.3, 0.3, e.nops)).cuda()
    E0, E1 = (torch.empty(1, dtype=torch.float64, device="cuda") for _ in range(2))
    g0, g1 = torch.empty_like(ang), torch.empty_like(ang)
    torch.cuda.synchronize()
    for v, y in zip(x, want):
        e.apply_dev(v.data_ptr(), y.data_ptr(), None, st[0].cuda_stream)
    e.gradient_dev(ang.data_ptr(), E0.data_ptr(), g0.data_ptr(), st[0].cuda_stream)
    torch.cuda.synchronize()
    for rep in range(20):
        got = [torch.empty_like(v) for v in x]
        torch.cuda.synchronize()
        for k in range(8):
            e.apply_dev(x[k % 4].data_ptr(), got[k % 4].data_ptr(), None, st[(k + rep) % 3].cuda_stream)
            if k == 3:
                e.gradient_dev(ang.data_ptr(), E1.data_ptr(), g1.data_ptr(), st[3].cuda_stream)
        torch.cuda.synchronize()
        for y, z in zip(got, want):
            assert torch.equal(y, z)
        assert torch.equal(E0, E1) and torch.equal(g0, g1)
    # a stream that is destroyed while its product may be in flight
    rt = torch.cuda.cudart()
    for rep in range(5):
        s = ctypes.c_void_p()
        assert int(rt.cudaStreamCreate(ctypes.addressof(s))) == 0
        e.apply_dev(x[0].data_ptr(), got[0].data_ptr(), None, s.value)
        assert int(rt.cudaStreamDestroy(s.value)) == 0
        e.apply_dev(x[1].data_ptr(), got[1].data_ptr(), None, st[1].cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    e.close()


@pytest.mark.parametrize("N,na,nb", [(10, 5, 4), (8, 4, 4)])
def test_recorded_by_the_caller(monkeypatch, N, na, nb):
    """The recorded product, energy and gradient are the FP64 kernels' (a replay may meet any
    other call); replays beside unrecorded products disturb neither."""
    e, ref = (make(monkeypatch, t, N, na, nb) for t in (True, False))
    rng = np.random.default_rng(N)
    x = torch.from_numpy(rng.standard_normal(e.D)).cuda()
    ang = torch.from_numpy(rng.uniform(-0.3, 0.3, e.nops)).cuda()
    y, z, w = (torch.empty_like(x) for _ in range(3))
    E = [torch.empty(1, dtype=torch.float64, device="cuda") for _ in range(3)]
    g, h = torch.empty_like(ang), torch.empty_like(ang)
    st, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for eng, out in ((e, w), (ref, z)):  # also loads every kernel before the recording
        eng.apply_dev(x.data_ptr(), out.data_ptr(), E[0].data_ptr(), st.cuda_stream)
    for eng in (e, ref):  # an engine's own graph cannot be recorded
        eng.use_graphs(False)
    ref.gradient_dev(ang.data_ptr(), E[2].data_ptr(), h.data_ptr(), st.cuda_stream)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        s = torch.cuda.current_stream().cuda_stream
        e.apply_dev(x.data_ptr(), y.data_ptr(), None, s)
        e.gradient_dev(ang.data_ptr(), E[1].data_ptr(), g.data_ptr(), s)
    got = torch.empty_like(x)
    for _ in range(10):
        y.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            graph.replay()
        for _ in range(4):
            e.apply_dev(x.data_ptr(), got.data_ptr(), None, other.cuda_stream)
        torch.cuda.synchronize()
        assert torch.equal(y, z) and torch.equal(got, w)
        assert torch.equal(E[1], E[2]) and torch.equal(g, h)
    e.close()
    ref.close()


def test_an_engine_twice_in_a_group(monkeypatch):
    """The evaluations of one engine in a group share its buffers: they run in turn."""
    a, b = (make(monkeypatch, True, 10, 5, 5) for _ in range(2))
    ang = np.random.default_rng(2).uniform(-0.3, 0.3, (2, a.nops))
    want = [a.gradient(ang[0]), b.gradient(ang[1])]
    group = ae.Group([a, b, a, a, b])
    for e, x in ((a, ang[0]), (b, ang[1])):
        e.io_put_angles(x)
    torch.cuda.synchronize()
    for _ in range(20):
        group.launch()
        group.sync()
        for e, (E, g) in ((a, want[0]), (b, want[1])):
            E1, g1 = e.io_get_results()
            assert np.array_equal(np.ravel(E1), np.ravel(E)) and np.array_equal(np.ravel(g1), np.ravel(g))
    group.close()
    a.close()
    b.close()
