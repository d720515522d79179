"""Class launches on side streams: builds from several threads and streams at
once, and a build captured by the caller (which stays on the caller's stream),
give the matrices of a build alone to the parity tolerance."""
import threading

import numpy as np
import pytest

from openlowdin_gb300 import systems as S

pytestmark = pytest.mark.gpu

TOL_FOCK = 1e-10


@pytest.fixture(scope="module")
def L():
    from openlowdin_gb300 import build, lint
    build.build()
    return lint


def _case(L, seed, o_d):
    torch = pytest.importorskip("torch")
    sp = S.water_cluster(2, seed=seed, o_d=o_d)["species"][0]
    h = L.Libint2Interface(sp, 1)
    X = np.random.default_rng(seed).normal(size=(h.nbasis, h.nbasis)) * 0.1
    D = torch.tensor(X + X.T, device="cuda")
    return h, D, torch.full_like(D, float("nan"))


@pytest.mark.parametrize("precision", [0, 1])
def test_builds_from_threads_match_builds_alone(L, precision):
    torch = pytest.importorskip("torch")
    cases = [_case(L, k, o_d=k % 2 == 0) for k in range(6)]
    split = 1e-5 if precision else 0.0
    alone = []
    for h, D, G in cases:
        h.twobody_device(D.data_ptr(), G.data_ptr(), -0.5, precision, split,
                         torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        alone.append(G.clone())
        G.fill_(float("nan"))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in cases]

    def work(k):
        h, D, G = cases[k]
        for _ in range(5):
            h.twobody_device(D.data_ptr(), G.data_ptr(), -0.5, precision, split, streams[k].cuda_stream)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(cases))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    tol = TOL_FOCK if precision == 0 else 1e-6
    for (h, _, G), ref in zip(cases, alone):
        assert float((G - ref).abs().max()) < tol * max(1.0, float(ref.abs().max()))
        h.close()


@pytest.mark.parametrize("o_d", [False, True])
def test_captured_build_matches_eager(L, o_d):
    torch = pytest.importorskip("torch")
    h, D, G = _case(L, 11, o_d)
    other, D2, G2 = _case(L, 12, o_d)

    def call(x, d, g, s):
        x.twobody_device(d.data_ptr(), g.data_ptr(), -0.5, stream=s.cuda_stream)

    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        call(h, D, G, st)
        call(other, D2, G2, st)
    torch.cuda.synchronize()
    ref, ref2 = G.clone(), G2.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st, capture_error_mode="thread_local"):
        call(h, D, G, torch.cuda.current_stream())
    G.fill_(float("nan"))
    G2.fill_(float("nan"))
    graph.replay()
    call(other, D2, G2, st)      # an eager build behind the capture
    torch.cuda.synchronize()
    assert float((G - ref).abs().max()) < TOL_FOCK * max(1.0, float(ref.abs().max()))
    assert float((G2 - ref2).abs().max()) < TOL_FOCK * max(1.0, float(ref2.abs().max()))
    h.close()
    other.close()
