"""The Gram kernel with more panel pairs than a grid's second dimension holds (a Hessian of more
than 23,103 parameters): two rows of whole numbers, so that every product and sum is exact."""
import numpy as np
import pytest

import ansatzevolve_gb300 as ae

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [23104, 23170])  # 361 panels: 65,341 pairs; 363 panels: 66,066
def test_many_columns(V):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(V)
    a, b = (torch.randint(-50, 50, (V, 2), generator=g, device="cuda").double() for _ in range(2))
    C = torch.full((V, V), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = ae.lib().aegpu_gram_upper_dev(a.data_ptr(), 2, b.data_ptr(), 2, 2, 1, V, 0.5, C.data_ptr(), None, V,
                                       torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    for j0 in range(0, V, 4096):  # column-major: C[j, i] = 0.5 a_i . b_j, i <= j
        c = C[j0:j0 + 4096]
        want = 0.5 * (b[j0:j0 + 4096] @ a.T)
        i, j = torch.arange(V, device="cuda"), torch.arange(j0, j0 + c.shape[0], device="cuda")
        on = i[None, :] <= j[:, None]
        assert torch.equal(c[on], want[on])
        assert torch.isnan(c[~on]).all()
