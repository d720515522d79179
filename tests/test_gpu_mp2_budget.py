"""MP2 whose column budget is below one pair of f shells (100 columns): the
batches then hold one pair each, and the energy is that of one batch."""
import numpy as np
import pytest

from openlowdin_gb300 import systems as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(0, 1e-12), (2, 1e-6)])
def test_budget_below_one_pair(precision, tol):
    torch = pytest.importorskip("torch")
    from openlowdin_gb300 import build, lint
    build.build()
    A, B = [0.0, 0.0, 0.0], [0.0, 0.9, 1.3]
    shells = [x for c in (A, B) for x in ((0, [0.8], [1.0], c), (1, [1.1], [1.0], c), (3, [1.3], [1.0], c))]
    h = lint.Libint2Interface(S.electron_species(shells, 6), 1)
    n, nocc = h.nbasis, 3
    rng = np.random.default_rng(4)
    C = rng.normal(size=(n, n)) * 0.2
    eps = np.concatenate([-3.0 + np.arange(nocc), 1.0 + np.arange(n - nocc)])
    dD, dC = torch.tensor(2.0 * C[:nocc].T @ C[:nocc], device="cuda"), torch.tensor(C, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    e = [h.mp2_direct(dD.data_ptr(), dC.data_ptr(), eps, nocc, 0, precision, gb, stream=st) for gb in (0.0, 1e-6)]
    h.close()
    assert e[0] < 0.0
    assert abs(e[1] - e[0]) <= tol * abs(e[0])
