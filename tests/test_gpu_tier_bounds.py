"""Where J/K builds leave FP64 for double-float arithmetic, element by element:
densities with one non-zero element, so that an element of the matrix is the
sum of two or three integrals, against the entry point that knows only FP64.

A double-float integral is within 2^-40 of its quartet's bound (2^-41.3 the
worst of six million of them), the tier ends at 2^-6 (plain builds, and mixed
ones with a small split), and both entry points evaluate the FP64 quartets with
the same kernels: two or three additions in another order, 2^-50 of their sum.
So an element differs by less than 3 * 2^-46 plus 2^-50 of the terms' size.
Without the tier's ends (or with the wrong side of them in double-float) large
elements differ by 2^-42 of themselves."""
import numpy as np
import pytest

from openlowdin_gb300 import systems as S

pytestmark = pytest.mark.gpu

DD = 3 * 2.0 ** -46


@pytest.fixture(scope="module")
def L():
    from openlowdin_gb300 import build, lint
    build.build()
    return lint


def _species(which):
    if which == "protons":
        return S.water_cluster(12, seed=3, quantum_protons=True, proton_species_mode="single")["species"][1]
    if which == "water_d":
        return S.water_cluster(8, seed=2, o_d=True)["species"][0]
    if which == "tight":
        # core functions of large exponent beside diffuse ones: a largest bound of
        # hundreds per density element
        rng = np.random.default_rng(8)
        shells = []
        for _ in range(10):
            o = list(rng.normal(size=3) * 3)
            shells += [(0, [a], [1.0], o) for a in (4.1e5, 9.7e3, 310.0, 12.0, 1.1, 0.13)]
            shells += [(1, [a], [1.0], o) for a in (5.2e2, 14.0, 0.9, 0.11)]
        return S.electron_species(shells, 20)
    return S.chain_for_basis(10_011, int(which))["species"][0]


class _Case:
    def __init__(self, L, sp):
        self.L, self.h, self.n = L, L.Libint2Interface(sp, 1), S.nbasis(sp)
        self.h.init_2body_ints()

    def builds(self, D, factor, precision=0, split=0.0):
        import torch
        st = torch.cuda.current_stream().cuda_stream
        d = torch.tensor(D, device="cuda")
        G, R = torch.full_like(d, float("nan")), torch.full_like(d, float("nan"))
        self.h.twobody_device(d.data_ptr(), G.data_ptr(), factor, precision, split, st)
        assert self.L.lib().LowdinGB300_twobody_device_noalloc(self.h.h, d.data_ptr(), R.data_ptr(), factor, 0, 0.0,
                                                               st) == 0
        torch.cuda.synchronize()
        return G.cpu().numpy(), R.cpu().numpy()

    def one(self, k, size, factor, **kw):
        D = np.zeros((self.n, self.n))
        D[k, k] = size
        return self.builds(D, factor, **kw)


def _functions(n):
    return np.random.default_rng(n).choice(n, 10, replace=False)


@pytest.mark.parametrize("which", ["240", "water_d", "tight"])
@pytest.mark.parametrize("size", [1.0, 40.0])
@pytest.mark.parametrize("split", [0.0, 1e-12])
def test_tier_ends(L, which, size, split):
    pytest.importorskip("torch")
    c = _Case(L, _species(which))
    entered = False
    for k in _functions(c.n):
        # Coulomb and exchange apart: no cancellation hides a term's size
        for factor in (0.0, -0.5):
            G, R = c.one(k, size, factor, precision=int(split > 0), split=split)
            diff = np.abs(G - R)
            J = np.abs(R if factor == 0.0 else c.one(k, size, 0.0)[1])
            assert np.all(diff <= DD + 2.0 ** -50 * (np.abs(R) + 2 * J)), (k, factor, float(diff.max()))
            # FP64 alone differs by less: the tier was entered
            entered |= bool(np.any(diff > 2.0 ** -49 * (np.abs(R) + 2 * J) + 1e-300))
    assert entered
    c.h.close()


@pytest.mark.parametrize("split", [0.0, 1e-12])
def test_tier_of_fp64_builds(L, oracle, split):
    # Coulomb alone: an element is one integral, not above its quartet's bound, and in
    # FP64 from 2^-12 of the largest bound on, also in mixed builds of a small split
    pytest.importorskip("torch")
    sp = _species("240")
    c = _Case(L, sp)
    tier = float(np.max(oracle.schwarz(oracle.Basis.from_shells(sp["shells"])))) ** 2 / 4096
    seen = 0
    for k in _functions(c.n):
        G, R = c.one(k, 1.0, 0.0, precision=int(split > 0), split=split)
        m = (np.abs(R) > 1.01 * tier) & (np.abs(R) < 2.0 ** -6)
        seen += int(m.sum())
        assert np.all(np.abs(G - R)[m] <= 2.0 ** -49 * np.abs(R[m]))
    assert seen > 100
    c.h.close()


def test_mixed_tier_stays_below_the_fp32_quartets(L):
    # split 1e-5: an FP32 integral is within some 2^-17 of its bound
    pytest.importorskip("torch")
    c = _Case(L, _species("240"))
    for k in _functions(c.n):
        G, R = c.one(k, 1.0, -0.5, precision=1, split=1e-5)
        assert np.max(np.abs(G - R)) <= 3e-5 * 2.0 ** -17
    c.h.close()


def test_unscreened_species_keep_fp64(L):
    # every element to the relative precision of its own integral, however small
    pytest.importorskip("torch")
    c = _Case(L, _species("protons"))
    for k in _functions(c.n):
        G, R = c.one(k, 1.0, 0.0)
        assert np.all(np.abs(G - R) <= 2.0 ** -49 * np.abs(R))
    c.h.close()


@pytest.mark.parametrize("scale", [1e12, 1e-9])
def test_contractions_of_another_scale(L, scale):
    # unnormalised contraction coefficients: the matrix in normalised functions is the same
    pytest.importorskip("torch")
    sp = _species("110")
    sp["shells"] = [(l, a, [scale * x for x in w], o) for l, a, w, o in sp["shells"]]
    c = _Case(L, sp)
    X = np.random.default_rng(3).normal(size=(c.n, c.n)) * 0.1
    G, R = c.builds(X + X.T, -0.5)
    assert np.all(np.isfinite(R))
    assert np.max(np.abs(G - R)) <= 1e-13 * np.max(np.abs(R))
    c.h.close()
