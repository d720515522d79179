"""Builds on independent streams do not wait for one another: a build or a
transform queued behind long work on one stream leaves builds on every other
stream free to finish.  And builds queued one behind another on one stream read
the density that is there when their turn comes, although their own launches
overlap."""
import threading
import time

import numpy as np
import pytest

from openlowdin_gb300 import systems as S

pytestmark = pytest.mark.gpu

HOLD = 500_000_000     # clock cycles: 0.25 s


@pytest.fixture(scope="module")
def L():
    from openlowdin_gb300 import build, lint
    build.build()
    return lint


class _Build:
    def __init__(self, L, seed):
        import torch
        self.h = L.Libint2Interface(S.water_cluster(1, seed=seed, place=False)["species"][0], 1)
        X = np.random.default_rng(seed).normal(size=(self.h.nbasis, self.h.nbasis)) * 0.1
        self.D = torch.tensor(X + X.T, device="cuda")
        self.G = torch.empty_like(self.D)
        self.s = torch.cuda.Stream()
        self.queue()
        torch.cuda.synchronize()
        self.ref = self.G.clone()
        self.G.fill_(float("nan"))
        torch.cuda.synchronize()

    def queue(self):
        self.h.twobody_device(self.D.data_ptr(), self.G.data_ptr(), -0.5, stream=self.s.cuda_stream)

    def hold(self):
        import torch
        with torch.cuda.stream(self.s):
            torch.cuda._sleep(HOLD)

    def done(self):
        return self.s.query()

    def right(self):
        return float((self.G - self.ref).abs().max()) < 1e-10 * max(1.0, float(self.ref.abs().max()))


def _finishes_first(free, held):
    """Whether stream `free` runs dry while every stream of `held` is still held."""
    t = time.perf_counter()
    while not free.done() and time.perf_counter() - t < 5.0:
        time.sleep(1e-3)
    return free.done() and not any(h.done() for h in held)


def test_build_does_not_wait_for_another_stream(L):
    torch = pytest.importorskip("torch")
    builds = [_Build(L, k) for k in range(5)]
    waited = []
    for a in builds:
        for b in builds:
            if a is b:
                continue
            a.hold()
            a.queue()
            b.queue()
            if not _finishes_first(b, [a]):
                waited.append((builds.index(a), builds.index(b)))
            torch.cuda.synchronize()
            assert a.right() and b.right()
    assert not waited


def test_build_does_not_wait_for_a_transform(L):
    torch = pytest.importorskip("torch")
    a, b = _Build(L, 3), _Build(L, 4)
    n, nocc = a.h.nbasis, 5
    rng = np.random.default_rng(5)
    C = torch.tensor(rng.normal(size=(n, n)) * 0.3, device="cuda")
    eps = np.concatenate([np.sort(-rng.uniform(0.5, 20.0, size=nocc)), np.sort(rng.uniform(0.1, 5.0, size=n - nocc))])

    def transform():
        # a small budget: several column batches, one behind the other
        a.h.mp2_direct(a.D.data_ptr(), C.data_ptr(), eps, nocc, 0, 0, 1e-4, stream=a.s.cuda_stream)

    transform()
    torch.cuda.synchronize()
    for _ in range(4):
        a.hold()
    t = threading.Thread(target=transform)
    t.start()
    time.sleep(0.1)      # its launches are queued, and it waits for the result
    b.queue()
    first = _finishes_first(b, [a])
    t.join()
    assert first
    torch.cuda.synchronize()
    assert b.right()


def test_many_streams_at_once(L):
    torch = pytest.importorskip("torch")
    builds = [_Build(L, 10 + k) for k in range(20)]
    for _ in range(3):
        for x in builds:
            x.queue()
    torch.cuda.synchronize()
    assert all(x.right() for x in builds)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("o_d", [False, True])
def test_queued_builds_read_their_own_density(L, precision, o_d):
    torch = pytest.importorskip("torch")
    h = L.Libint2Interface(S.water_cluster(2, seed=7, o_d=o_d)["species"][0], 1)
    n, st = h.nbasis, torch.cuda.current_stream()
    rng = np.random.default_rng(9)
    X = [rng.normal(size=(n, n)) * 10.0 ** -k for k in range(6)]
    dens = [torch.tensor(x + x.T, device="cuda") for x in X]
    D = torch.empty_like(dens[0])
    split = 1e-5 if precision else 0.0

    def build(d, g):
        D.copy_(d)
        h.twobody_device(D.data_ptr(), g.data_ptr(), -0.5, precision, split, st.cuda_stream)

    alone = [torch.empty_like(D) for _ in dens]
    for d, g in zip(dens, alone):
        build(d, g)
        torch.cuda.synchronize()
    order = [k for _ in range(10) for k in rng.permutation(len(dens))]
    queued = [torch.full_like(D, float("nan")) for _ in order]
    for k, g in zip(order, queued):
        build(dens[k], g)
    torch.cuda.synchronize()
    tol = 1e-12 if precision == 0 else 1e-6
    for k, g in zip(order, queued):
        assert float((g - alone[k]).abs().max()) <= tol * float(alone[k].abs().max())
    h.close()
