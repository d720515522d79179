"""Contracted shells on the kernels that deal a quartet's primitive quartets to
several lanes and slices: every direct entry against the oracle, with
contractions of 1 to 9 primitives (remainders of every lane count), classes up
to (dd|dd), one and two centres.  Tolerances of the parity tests: 1e-10 on
matrices, 1e-9 on first-quarter tensors (absolute, elements of order one)."""
import numpy as np
import pytest

from openlowdin_gb300 import systems as S

pytestmark = pytest.mark.gpu

TOL_FOCK, TOL_IT = 1e-10, 1e-9


@pytest.fixture(scope="module")
def L():
    from openlowdin_gb300 import build, lint
    build.build()
    return lint


def _shells(which):
    rng = np.random.default_rng(17)

    def con(lo, ratio, k):
        return [lo * ratio ** (k - 1 - i) for i in range(k)], list(rng.uniform(0.2, 1.0, size=k))

    centres = [[0.0, 0.0, 0.0], [0.4, -1.3, 1.1], [-1.2, 0.8, 1.9]]
    spec = {"s9": [(0, 9), (0, 1)], "sp": [(0, 6), (0, 3), (1, 5), (1, 1)],
            "spd": [(0, 7), (1, 3), (2, 2), (2, 1)]}[which]
    out = []
    for c in centres[: 2 if which == "spd" else 3]:
        for l, k in spec:
            a, w = con(0.25 + 0.1 * l, 2.7, k)
            out.append((l, a, w, c))
    return out


def _dens(n, seed):
    X = np.random.default_rng(seed).normal(size=(n, n)) * 0.2
    return X + X.T


@pytest.mark.parametrize("which", ["s9", "sp", "spd"])
def test_contracted_two_body(L, oracle, which):
    sp = S.electron_species(_shells(which), 4)
    n = S.nbasis(sp)
    D = _dens(n, 1)
    h = L.Libint2Interface(sp, 1)
    b = oracle.Basis.from_shells(sp["shells"])
    G = h.compute_2body_direct(D, -0.5)
    ref = oracle.two_body_direct(b, True, D, -0.5)
    assert np.max(np.abs(G - ref)) < TOL_FOCK * max(1.0, np.max(np.abs(ref)))
    assert h.last_quartets() == oracle.last_quartet_count()
    C = np.random.default_rng(2).normal(size=(n, n))
    A = h.compute_2body_directIT(D, C, n - 1)
    assert np.max(np.abs(A - oracle.two_body_directIT(b, True, D, C, n - 1))) < TOL_IT
    g, c = [0.7, 3.1], [0.4, -0.2]
    G = h.compute_g12_direct(D, -0.5, c, g)
    ref = oracle.g12_direct(b, D, -0.5, c, g)
    assert np.max(np.abs(G - ref)) < TOL_FOCK * max(1.0, np.max(np.abs(ref)))
    h.close()


@pytest.mark.parametrize("which", ["s9", "sp", "spd"])
def test_contracted_coupling(L, oracle, which):
    e = S.electron_species(_shells(which), 4)
    p = S.proton_species([(0, [4.0, 9.0, 21.0], [0.5, 0.4, 0.3], [0.4, -1.3, 1.1]),
                          (1, [7.0, 16.0], [0.6, 0.5], [0.4, -1.3, 1.1])], 1)
    he, hp = L.Libint2Interface(e, 1), L.Libint2Interface(p, 2)
    be, bp = (oracle.Basis.from_shells(x["shells"]) for x in (e, p))
    for A, ia, ba, B, ib, bb in ((he, 1, be, hp, 2, bp), (hp, 2, bp, he, 1, be)):
        D = _dens(B.nbasis, 3)
        assert np.max(np.abs(A.compute_coupling_direct(B, D) - oracle.coupling_direct(ba, ia, bb, ib, D))) < TOL_FOCK
        got = A.compute_g12inter_direct(B, D, [0.4, -0.2], [0.7, 3.1])
        ref = oracle.g12inter_direct(ba, ia, bb, ib, D, [0.4, -0.2], [0.7, 3.1])
        assert np.max(np.abs(got - ref)) < TOL_FOCK
    he.close()
    hp.close()
