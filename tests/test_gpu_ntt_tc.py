"""The tensor-core NTT passes against the CPU oracle, bit for bit: the smallest transform that
takes them and the one below it, each tile size, ragged splits of the layers over the passes, the
layers whose 128-butterfly tiles hold one, two, four and more twiddles, and data whose bit counts
are the largest a product can sum (elements of all ones against all-ones twiddle rows)."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA device", allow_module_level=True)

import binius64_b200 as bg  # noqa: E402


@pytest.mark.parametrize("ones", [False, True])
@pytest.mark.parametrize("log_d,skip_early,skip_late", [
    (10, 0, 0), (11, 0, 0), (11, 1, 0), (11, 2, 3), (12, 0, 6), (13, 2, 5), (17, 0, 1),
    (18, 0, 0), (18, 7, 4), (18, 8, 4), (19, 1, 7), (20, 3, 2), (21, 0, 9),
])
def test_transforms(log_d, skip_early, skip_late, ones):
    r = np.random.default_rng(log_d * 100 + skip_early * 10 + skip_late)
    data = orc.random_elems(r, 1 << log_d)
    if ones:  # the upper elements of the first inverse layer's pairs, the lower ones zero
        upper = (np.arange(1 << log_d) >> skip_late) & 1
        data = np.repeat((upper.astype(np.uint64) * np.uint64(2**64 - 1))[:, None], 2, axis=1)
    ntt = bg.AdditiveNTT(log_d)
    tw = orc.domain_twiddles(log_d)
    d = bg.to_device(data)
    ntt.forward_transform(d, skip_early, skip_late)
    ref = orc.ntt_forward(tw, log_d, data, skip_early, skip_late)
    assert np.array_equal(bg.to_host(d), ref)
    ntt.inverse_transform(d, skip_early, skip_late)
    assert np.array_equal(bg.to_host(d), data)
    ntt.inverse_transform(d, skip_early, skip_late)
    ntt.forward_transform(d, skip_early, skip_late)
    assert np.array_equal(bg.to_host(d), data)


@pytest.mark.parametrize("log_dim,log_inv_rate,log_batch", [
    (9, 1, 0), (9, 2, 0), (4, 1, 6), (7, 3, 1), (13, 1, 4), (11, 2, 5), (12, 2, 7), (19, 1, 0),
])
def test_encode(log_dim, log_inv_rate, log_batch):
    r = np.random.default_rng(300 + log_dim)
    n = log_dim + log_inv_rate
    basis = bg.standard_domain_rs_basis(n + log_batch, log_batch)
    tw = orc.domain_twiddles(n, basis=basis)
    msg = orc.random_elems(r, 1 << (log_dim + log_batch))
    out = bg.ReedSolomonCode(log_dim, log_inv_rate).encode_batch(
        bg.AdditiveNTT(n, basis=basis), bg.to_device(msg), log_batch)
    assert np.array_equal(bg.to_host(out),
                          orc.rs_encode_batch(tw, n, msg, log_dim, log_inv_rate, log_batch))


@pytest.mark.parametrize("log_d,skip_early,skip_late", [
    (10, 0, 1), (11, 1, 1), (11, 0, 1), (12, 2, 0), (12, 1, 0), (14, 4, 3), (15, 5, 0), (15, 4, 0),
    (16, 6, 0), (16, 7, 0), (17, 7, 1),
])
def test_transforms_where_the_passes_change(log_d, skip_early, skip_late):
    """Butterflies within ten index bits and eleven, on either side of the size from which ten take
    the tensor-core passes, with the encode of the same layers where there is one."""
    r = np.random.default_rng(5000 + log_d * 100 + skip_early * 10 + skip_late)
    data = orc.random_elems(r, 1 << log_d)
    ntt = bg.AdditiveNTT(log_d)
    tw = orc.domain_twiddles(log_d)
    d = bg.to_device(data)
    ntt.forward_transform(d, skip_early, skip_late)
    assert np.array_equal(bg.to_host(d), orc.ntt_forward(tw, log_d, data, skip_early, skip_late))
    ntt.inverse_transform(d, skip_early, skip_late)
    assert np.array_equal(bg.to_host(d), data)
    if 1 <= skip_early <= 4:
        n, dim = log_d - skip_late, log_d - skip_late - skip_early
        basis = bg.standard_domain_rs_basis(log_d, skip_late)
        tw = orc.domain_twiddles(n, basis=basis)
        msg = data[:1 << (log_d - skip_early)]
        out = bg.ReedSolomonCode(dim, skip_early).encode_batch(
            bg.AdditiveNTT(n, basis=basis), bg.to_device(msg), skip_late)
        assert np.array_equal(bg.to_host(out),
                              orc.rs_encode_batch(tw, n, msg, dim, skip_early, skip_late))
