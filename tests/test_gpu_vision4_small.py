"""The four-warps-per-permutation Vision-4 trees against the oracle, node for node: one leaf and
no layer, odd numbers of layers above the fused ones, the sizes where the leaves per CTA change and
where the one-thread kernels take over, long sponges, and leaves whose first sbox sees zeros."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA device", allow_module_level=True)

import binius64_b200 as bg  # noqa: E402


@pytest.mark.parametrize("log_leaves,log_batch", [
    (0, 7), (1, 1), (2, 0), (4, 5), (5, 3), (6, 7), (7, 1), (8, 1), (9, 0), (11, 1), (12, 1), (13, 0),
])
def test_commit(log_leaves, log_batch):
    r = np.random.default_rng(900 + 8 * log_leaves + log_batch)
    elems = orc.random_elems(r, 1 << (log_leaves + log_batch))
    rc, _ = orc.vision4_constants()
    elems[0] = orc.from_int(rc[0][0])  # a zero enters the first sbox of leaf 0
    if log_batch:
        elems[1] = orc.from_int(rc[0][1])
        elems[-1] = 0
    orc.set_threads(8)
    try:
        ref = orc.vision4_merkle_commit(elems, log_leaves, log_batch)
    finally:
        orc.set_threads(1)
    root, committed = bg.BinaryMerkleTreeProver("vision4").commit(bg.to_device(elems),
                                                                  1 << log_batch)
    assert np.array_equal(committed.nodes.cpu().numpy(), ref)
    assert root == bytes(ref[-1])
