"""A batch of more species than a grid has rows (65,535): every system of it is
built.  The systems share one handle of two s functions and differ in their
densities; reference: the oracle's matrix, linear in the density."""
import numpy as np
import pytest

from openlowdin_gb300 import systems as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L():
    from openlowdin_gb300 import build, lint
    build.build()
    return lint


@pytest.mark.parametrize("count", [65_535, 65_600])
def test_many_species(L, oracle, count):
    torch = pytest.importorskip("torch")
    sp = S.electron_species([(0, [1.3], [1.0], [0.0, 0.0, 0.0]), (0, [0.4], [1.0], [0.0, 0.3, 0.9])], 2)
    h = L.Libint2Interface(sp, 1)
    st = torch.cuda.current_stream().cuda_stream
    scale = torch.linspace(0.5, 1.5, count, dtype=torch.float64, device="cuda")
    D = np.array([[0.7, -0.2], [-0.2, 0.4]])
    P = scale[:, None, None] * torch.tensor(D, device="cuda")
    G, J = torch.full_like(P, float("nan")), torch.full_like(P, float("nan"))
    b = L.Batch()
    for k in range(count):
        at = 32 * k
        b.add_system([h], [-1.0], [-0.5], [1], [P.data_ptr() + at], [G.data_ptr() + at], [J.data_ptr() + at])
    b.finalize(st)
    b.fock(0, 0.0, st)
    torch.cuda.synchronize()
    ref = torch.tensor(oracle.two_body_direct(oracle.Basis.from_shells(sp["shells"]), True, D, -0.5), device="cuda")
    assert float((G - scale[:, None, None] * ref).abs().max()) < 1e-10
    b.close()
    h.close()
