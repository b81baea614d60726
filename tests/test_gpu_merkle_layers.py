"""SHA-256 trees against the CPU oracle, every digest: the sizes around those where another kernel or
another split of the layers over the launches begins, and leaves of one element, two, one block and
several, whose last blocks are formed differently by each kernel."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA device", allow_module_level=True)

import binius64_b200 as bg  # noqa: E402


@pytest.mark.parametrize("log_leaves,log_batch", [
    (0, 0), (0, 3), (1, 7), (2, 2), (3, 1), (4, 4), (5, 0), (6, 3), (8, 4), (9, 2), (11, 0), (12, 1),
    (13, 2), (14, 0), (16, 0), (17, 0), (17, 1), (18, 2), (19, 0), (20, 1), (17, 3), (7, 7),
])
def test_trees(log_leaves, log_batch):
    r = np.random.default_rng(10 * log_leaves + log_batch)
    elems = orc.random_elems(r, 1 << (log_leaves + log_batch))
    root, tree = bg.BinaryMerkleTreeProver().commit(bg.to_device(elems), 1 << log_batch)
    ref = orc.merkle_commit(elems, log_leaves, log_batch)
    assert np.array_equal(tree.nodes.cpu().numpy(), ref.reshape(-1, 32))
    assert root == ref.reshape(-1, 32)[-1].tobytes()
