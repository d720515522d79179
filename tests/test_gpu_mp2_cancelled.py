"""Split-BF16 MP2 on an integral that its own terms cancel down to the 1e-10 cut:
an s and a p function on two centres, and two s functions of another species
beside the root of (s p|s s) along their axis.  With these bases the inter-species
term is f (s p|s s)^2 / (energies), so it shows the one integral to relative
precision, and whether it passed the cut.

The integral is a sum of two products of 0.1, each within 2^-46 of itself in
double-float; the split form rounds it and the coefficients to 24 bits: six
roundings, and the square has twice the relative error."""
import numpy as np
import pytest

from openlowdin_gb300 import systems as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L():
    from openlowdin_gb300 import build, lint
    build.build()
    return lint


def _shells(c):
    return ([(0, [0.2], [1.0], [0.0, 0.0, 0.0]), (1, [3.0], [1.0], [0.0, 0.0, 1.4])],
            [(0, [1.1], [1.0], [0.0, 0.0, c]), (0, [2.3], [1.0], [0.0, 0.0, c])])


@pytest.mark.parametrize("target", [0.999e-10, 1.001e-10, 2e-10, -3e-9])
def test_cancelled_integral(L, oracle, target):
    torch = pytest.importorskip("torch")

    def integral(c):
        a, b = _shells(c)
        return oracle.eri_quartet(oracle.Basis.from_shells(a + b), 0, 1, 2, 3).ravel()[2]   # (s pz|s s)

    lo, hi = 1.2, 2.0
    assert integral(lo) * integral(hi) < 0
    sign = np.sign(integral(hi))
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        if sign * (integral(mid) - target) > 0:
            hi = mid
        else:
            lo = mid
    a, b = _shells(hi)
    assert abs(integral(hi) - target) < 1e-4 * abs(target)
    A = L.Libint2Interface(S.electron_species(a, 2), 1)
    B = L.Libint2Interface(S.proton_species(b, 1), 2)
    CA, CB = torch.eye(4, dtype=torch.float64, device="cuda"), torch.eye(2, dtype=torch.float64, device="cuda")
    ea, eb = np.array([-1.0, 1.0, 1.1, 1.2]), np.array([-0.5, 0.7])
    st = torch.cuda.current_stream().cuda_stream

    def term(precision):
        # a factor that lifts the square out of the far end of the range
        return A.mp2_coupling(B, CA.data_ptr(), CB.data_ptr(), ea, eb, 1, 0, 1, 0, 1e18, precision, stream=st)

    exact, split = term(0), term(2)
    if abs(target) < 1e-10:
        assert exact == 0.0 and split == 0.0
    else:
        assert exact != 0.0
        assert abs(split / exact - 1.0) < 2 * (6 * 2.0 ** -24 + 2 * 0.1 * 2.0 ** -46 / abs(target))
    A.close()
    B.close()
