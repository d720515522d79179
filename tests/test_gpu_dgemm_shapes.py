"""FP64 MP2 transform at the edges of its matrix tiles: occupied and virtual
counts around multiples of 8 and 64, odd basis sizes (remainders of the
instruction's k of 4), against the transform of the full integral tensor in
numpy (FP64).  Tolerance 1e-10 Eh as the other FP64 MP2 tests."""
import numpy as np
import pytest

from openlowdin_gb300 import systems as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L():
    from openlowdin_gb300 import build, lint
    build.build()
    return lint


@pytest.mark.parametrize("n_shells,nocc,frozen", [(13, 1, 0), (13, 7, 0), (13, 9, 1), (14, 8, 0), (15, 14, 2),
                                                  (9, 20, 3), (9, 2, 1)])
@pytest.mark.parametrize("budget", [0.0, 2e-4])
def test_fp64_transform_edges(L, oracle, n_shells, nocc, frozen, budget):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n_shells * 31 + nocc)
    shells = [(int(l), [float(a)], [1.0], list(rng.normal(size=3) * 1.5))
              for l, a in zip(rng.permutation([k % 3 if n_shells == 9 else k % 2 for k in range(n_shells)]),
                              rng.uniform(0.2, 6.0, size=n_shells))]
    sp = S.electron_species(shells, 2 * nocc)
    b = oracle.Basis.from_shells(shells)
    n = b.nbf
    assert nocc < n
    C = rng.normal(size=(n, n)) * 0.3
    eps = np.concatenate([np.sort(-rng.uniform(0.5, 20.0, size=nocc)), np.sort(rng.uniform(0.1, 5.0, size=n - nocc))])
    D = 2.0 * C[:nocc].T @ C[:nocc]
    h = L.Libint2Interface(sp, 1)
    dD, dC = torch.tensor(D, device="cuda"), torch.tensor(C, device="cuda")
    e2 = h.mp2_direct(dD.data_ptr(), dC.data_ptr(), eps, nocc, frozen, 0, budget,
                      stream=torch.cuda.current_stream().cuda_stream)
    h.close()
    eri = oracle.eri_full(b).reshape(n, n, n, n)
    o, v = C[frozen:nocc], C[nocc:]
    I = np.einsum("im,mnls->inls", o, eri, optimize=True)
    I = np.einsum("an,inls->ials", v, I, optimize=True)
    I = np.einsum("jl,ials->iajs", o, I, optimize=True)
    I = np.einsum("bs,iajs->iajb", v, I, optimize=True)
    gap = (eps[frozen:nocc, None, None, None] + eps[None, None, frozen:nocc, None]
           - eps[None, nocc:, None, None] - eps[None, None, None, nocc:])
    ref = float(np.sum(I * (2 * I - I.transpose(0, 3, 2, 1)) / gap))
    # the library drops raw integrals below 1e-10: at most that much per element
    # of the transform, |C|^4 sums of them in each of the squared integrals
    assert abs(e2 - ref) < 1e-10 * max(1.0, abs(ref)) + 1e-9 * np.sqrt(abs(ref)), (e2, ref)
