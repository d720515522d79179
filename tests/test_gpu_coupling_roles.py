"""Coupling builds, whose kets come from the species with more pairs of the
class: both orders of the species against the oracle (1e-10 of the parity
tests), one pair against hundreds as well as hundreds against hundreds."""
import numpy as np
import pytest

from openlowdin_gb300 import systems as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L():
    from openlowdin_gb300 import build, lint
    build.build()
    return lint


def _dens(n, seed):
    X = np.random.default_rng(seed).normal(size=(n, n)) * 0.2
    return X + X.T


@pytest.mark.parametrize("n_waters,mode", [(1, "per_proton"), (2, "single"), (4, "single")])
def test_coupling_matches_oracle(L, oracle, n_waters, mode):
    torch = pytest.importorskip("torch")
    st = torch.cuda.current_stream().cuda_stream
    m = S.water_cluster(n_waters, seed=5, quantum_protons=True, proton_species_mode=mode, place=n_waters > 1)
    e, p = m["species"][:2]
    he, hp = L.Libint2Interface(e, 1), L.Libint2Interface(p, 2)
    be, bp = (oracle.Basis.from_shells(x["shells"]) for x in (e, p))
    De, Dp = _dens(he.nbasis, 1), _dens(hp.nbasis, 2)
    re, rp = oracle.coupling_direct(be, 1, bp, 2, Dp), oracle.coupling_direct(bp, 2, be, 1, De)
    for a, b, Da, Db, ra, rb in ((he, hp, De, Dp, re, rp), (hp, he, Dp, De, rp, re)):
        da, db = torch.tensor(Da, device="cuda"), torch.tensor(Db, device="cuda")
        ja, jb = torch.full_like(da, float("nan")), torch.full_like(db, float("nan"))
        L.coupling_device(a, b, da.data_ptr(), db.data_ptr(), ja.data_ptr(), jb.data_ptr(), stream=st)
        torch.cuda.synchronize()
        for j, r in ((ja.cpu().numpy(), ra), (jb.cpu().numpy(), rb)):
            assert np.max(np.abs(np.tril(j) - r)) < 1e-10 * max(1.0, np.max(np.abs(r)))
            assert np.max(np.abs(j - j.T)) <= 1e-12 * max(1.0, np.max(np.abs(j)))
    he.close()
    hp.close()
