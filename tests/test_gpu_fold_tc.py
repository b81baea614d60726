"""FRI folds against the oracle: interleaved folds on the tensor cores (the smallest size that takes
them and the one below, one to 256 columns, so half a pair of weights up to sixteen passes, all-ones
columns with all-ones weights, whose counts are the largest a sum can hold), and codeword folds whose
host challenges include 0 and 1 (a round of challenge 1 has no scaling factor)."""
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


@pytest.mark.parametrize("kind", ["random", "ones", "zero_one"])
@pytest.mark.parametrize("log_len,log_batch", [
    (6, 4), (7, 1), (7, 4), (8, 2), (9, 3), (10, 5), (8, 8), (13, 4), (7, 0),
])
def test_fold_interleaved(log_len, log_batch, kind):
    r = np.random.default_rng(1000 + 10 * log_len + log_batch)
    cw = orc.random_elems(r, 1 << (log_len + log_batch))
    ch = orc.random_elems(r, log_batch)
    if kind == "ones":
        cw[:] = np.uint64(2**64 - 1)
        ch[:] = np.uint64(2**64 - 1)
    elif kind == "zero_one" and log_batch:
        ch[0] = orc.from_int(1)
        ch[-1] = orc.from_int(0)
    out = bg.fold_interleaved(bg.to_device(cw), ints(ch), log_len, log_batch)
    assert np.array_equal(bg.to_host(out), orc.fri_fold_interleaved(cw, log_len, log_batch, ch))


@pytest.mark.parametrize("log_len", [4, 12, 20])
@pytest.mark.parametrize("challenges", [[1], [0, 5], [1, 1, 1, 1], [7, 1, 0, 9], [3, 4, 1, 6, 1, 8]])
def test_fold_codeword(log_len, challenges):
    if len(challenges) > log_len:
        pytest.skip("more challenges than variables")
    r = np.random.default_rng(2000 + log_len)
    cw = orc.random_elems(r, 1 << log_len)
    ch = [c if c < 2 else orc.to_int(orc.random_elems(r, 1)[0]) for c in challenges]
    ntt = bg.AdditiveNTT(log_len)
    tw = orc.domain_twiddles(log_len)
    out = bg.fold_codeword(ntt, bg.to_device(cw), ch, log_len)
    ref = orc.fri_fold_codeword(tw, log_len, cw, log_len,
                                np.array([orc.from_int(c) for c in ch], dtype=np.uint64))
    assert np.array_equal(bg.to_host(out), ref)


@pytest.mark.parametrize("log_len", [15, 16, 17, 18])
@pytest.mark.parametrize("challenges", [[3], [4, 1], [5, 6], [7, 0, 1], [8, 9, 3], [1, 4, 5, 6],
                                        [7, 8, 9, 3, 4], [1, 5, 6, 7, 8, 9]])
def test_fold_codeword_where_the_form_changes(log_len, challenges):
    """Rounds of one product and of two, on either side of the sizes from which the first begin, for
    one to four challenges a launch."""
    r = np.random.default_rng(3000 + log_len)
    cw = orc.random_elems(r, 1 << log_len)
    ch = [c if c < 2 else orc.to_int(orc.random_elems(r, 1)[0]) for c in challenges]
    ntt = bg.AdditiveNTT(log_len)
    tw = orc.domain_twiddles(log_len)
    out = bg.fold_codeword(ntt, bg.to_device(cw), ch, log_len)
    ref = orc.fri_fold_codeword(tw, log_len, cw, log_len,
                                np.array([orc.from_int(c) for c in ch], dtype=np.uint64))
    assert np.array_equal(bg.to_host(out), ref)
