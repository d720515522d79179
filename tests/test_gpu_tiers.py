"""J/K builds in two tiers (FP64 above a bound, double-float below) against the
build that knows only FP64 (the allocation-free entry point), over densities of
very different size, several species kinds and sizes on both sides of the
tier's minimum.

Tolerance: a double-float quartet's error is below 2^-43 of its bound, the bound
below 2^-12 of the largest one B, and fewer than 2^16 of them meet in one
element, with random signs: 2^-47 B = 7e-15 B; the FP64 sums of both builds,
added in any order, differ by up to some 1e-14 of the largest element.  Both
together stay below 1e-13 of it.
"""
import numpy as np
import pytest

from openlowdin_gb300 import systems as S

pytestmark = pytest.mark.gpu

TOL = 1e-13


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
        # core functions of large exponent beside diffuse ones on other centres
        rng = np.random.default_rng(8)
        shells = []
        for _ in range(10):
            o = list(rng.normal(size=3) * 3)
            shells += [(0, [a], [1.0], o) for a in (4.1e5, 9.7e3, 310.0, 12.0, 1.1, 0.13)]
            shells += [(1, [a], [1.0], o) for a in (5.2e2, 14.0, 0.9, 0.11)]
        return S.electron_species(shells, 20)
    return S.chain_for_basis(10_011, int(which))["species"][0]


def _both(L, sp, D):
    torch = pytest.importorskip("torch")
    h = L.Libint2Interface(sp, 1)
    h.init_2body_ints()
    factor = -0.5 if sp["is_electron"] else -1.0
    st = torch.cuda.current_stream().cuda_stream
    d = torch.tensor(D, device="cuda")
    G, R = torch.full_like(d, float("nan")), torch.full_like(d, float("nan"))
    h.twobody_device(d.data_ptr(), G.data_ptr(), factor, stream=st)
    torch.cuda.synchronize()
    count = h.last_quartets()
    assert L.lib().LowdinGB300_twobody_device_noalloc(h.h, d.data_ptr(), R.data_ptr(), factor, 0, 0.0, st) == 0
    torch.cuda.synchronize()
    h.close()
    return G.cpu().numpy(), R.cpu().numpy(), count


@pytest.mark.parametrize("which", ["36", "110", "240", "protons", "water_d", "tight"])
@pytest.mark.parametrize("scale", [1.0, 1e-5, 1e-14, 1e18])
def test_tiers_match_fp64(L, which, scale):
    sp = _species(which)
    n = S.nbasis(sp)
    X = np.random.default_rng(n).normal(size=(n, n)) * 0.1
    X[: n // 2] *= 1e-3          # elements of different size
    G, R, _ = _both(L, sp, scale * (X + X.T))
    top = np.max(np.abs(R))
    assert np.all(np.isfinite(G))
    assert np.max(np.abs(G - R)) <= TOL * top


def test_tiers_keep_the_quartets(L, oracle):
    sp = _species("110")
    n = S.nbasis(sp)
    X = np.random.default_rng(5).normal(size=(n, n)) * 0.1
    D = X + X.T
    G, _, count = _both(L, sp, D)
    ref = oracle.two_body_direct(oracle.Basis.from_shells(sp["shells"]), True, D, -0.5)
    assert np.max(np.abs(G - ref)) < 1e-10 * max(1.0, np.max(np.abs(ref)))
    assert count == oracle.last_quartet_count()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_bad_density_elements_stay_in_fp64(L, bad):
    sp = _species("110")
    n = S.nbasis(sp)
    X = np.random.default_rng(6).normal(size=(n, n)) * 0.1
    D = X + X.T
    D[3, 7] = D[7, 3] = bad
    G, R, _ = _both(L, sp, D)
    assert np.array_equal(np.isfinite(G), np.isfinite(R))
