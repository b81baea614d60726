"""Bivariate rounds whose next sums are queued by fold(): against the oracle at the sizes where the
round kernels change, for provers that run in turn, one dropped with a round in flight, and more
provers alive than there are pinned result slots."""
import ctypes

import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA device", allow_module_level=True)

import binius64_b200 as bg  # noqa: E402


def ints(a):
    return [orc.to_int(x) for x in a]


def case(n, seed):
    r = np.random.default_rng(seed)
    a, b = orc.random_elems(r, 1 << n), orc.random_elems(r, 1 << n)
    s = orc.to_int(orc.random_elems(r, 1)[0])  # a claim the rounds need not be true to
    ch = orc.random_elems(r, n)
    co, fin = orc.bivariate_rounds(a, b, s, ch)
    return (bg.BivariateProductSumcheckProver(bg.to_device(a), bg.to_device(b), s), ints(ch),
            [ints(c) for c in co], ints(fin))


@pytest.mark.parametrize("n", [1, 2, 7, 13, 15, 16])
def test_rounds(n):
    p, ch, co, fin = case(n, 800 + n)
    for k, r in enumerate(ch):
        assert p.execute() == co[k]
        p.fold(r)
        assert p.n_vars() == n - 1 - k
    assert p.finish() == fin


def test_in_turn_and_dropped():
    ps = [case(n, 900 + n) for n in (9, 4, 6)]
    dropped = case(8, 950)
    assert dropped[0].execute() == dropped[2][0]
    dropped[0].fold(dropped[1][0])
    del dropped
    for k in range(9):
        for p, ch, co, fin in ps:
            if k < len(ch):
                assert p.execute() == co[k]
                p.fold(ch[k])
    for p, _, _, fin in ps:
        assert p.finish() == fin


def test_more_provers_than_slots():
    a = bg.to_device(orc.random_elems(np.random.default_rng(1), 2))
    held = [bg.BivariateProductSumcheckProver(a, a, 0) for _ in range(1030)]
    p, ch, co, fin = case(5, 977)
    for k, r in enumerate(ch):
        assert p.execute() == co[k]
        p.fold(r)
    assert p.finish() == fin
    del held


@pytest.mark.parametrize("kind,n", [("bivariate", 1), ("bivariate", 9), ("quadratic", 6),
                                    ("inout", 5)])
def test_destroy_waits_on_the_default_stream(kind, n):
    """A prover on the legacy default stream that is dropped with a fold still queued: its multilinears
    are the caller's again when the drop returns."""
    r = np.random.default_rng(40 + n)
    elems = [bg.to_device(orc.random_elems(r, 1 << n)) for _ in range(3)]
    point = ints(orc.random_elems(r, n))
    if kind == "bivariate":
        p = bg.BivariateProductSumcheckProver(*elems[:2], 3)
    elif kind == "quadratic":
        p = bg.QuadraticMleCheckProver(*elems, point, 3)
    else:
        p = bg.InOutCheckProver(elems[0], point[:3])
    s = torch.cuda.default_stream()
    assert torch.cuda.current_stream() == s and s.cuda_stream == 0
    p.execute()
    torch.cuda._sleep(100_000_000)  # some 50 ms of the stream ahead of the fold
    p.fold(7)
    assert not s.query()
    del p
    assert s.query()


@pytest.mark.parametrize("n", [3, 9, 16])
def test_fold_that_fails_leaves_the_prover_as_it_was(n):
    """A fold whose launches are refused (its stream records a capture that has been invalidated by a
    synchronisation, which CUDA answers with an error) can be called again afterwards."""
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        p, ch, co, fin = case(n, 700 + n)
        assert p.execute() == co[0]
        p.fold(ch[0])
        assert p.execute() == co[1]
        s.synchronize()
        rt = ctypes.CDLL("libcudart.so.12")  # the one torch has loaded
        stream, graph = ctypes.c_void_p(s.cuda_stream), ctypes.c_void_p()
        assert rt.cudaStreamBeginCapture(stream, 2) == 0
        try:
            assert rt.cudaStreamSynchronize(stream) != 0
            for _ in range(2):
                with pytest.raises(bg.BiniusError):
                    p.fold(ch[1])
                assert p.n_vars() == n - 1
        finally:
            assert rt.cudaStreamEndCapture(stream, ctypes.byref(graph)) != 0
        rt.cudaGetLastError()
        for k in range(1, n):
            p.fold(ch[k])
            if k + 1 < n:
                assert p.execute() == co[k + 1]
        assert p.finish() == fin
