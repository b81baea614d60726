"""The shift reduction's in/out check against the oracle where its dot products go with the folds of
the launched rounds: public segments of one word pair, of a part and of half of the words (rounds
before, at and past the segment), below and above the folds' two sizes of kernel."""
import numpy as np
import pytest

import oracle as orc
from binius64_b200 import constraint_system as csm

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA device", allow_module_level=True)

import binius64_b200 as bg  # noqa: E402
from test_gpu_shift import _ints, _operator_data  # noqa: E402


@pytest.mark.parametrize("log_words,n_and,log_public", [
    (12, 1000, 11), (13, 2000, 1), (13, 2000, 12), (14, 5000, 12), (17, 30000, 14), (17, 30000, 16),
])
def test_public_segments(log_words, n_and, log_public):
    sc = csm.synthetic_circuit(log_words, n_and, 3, seed=log_words, log_public=log_public)
    prep, band, bmul = _operator_data(sc, seed=log_words)
    proof, point, out3 = orc.shift_prove(sc.witness, log_public, prep.and_csr, prep.mul_csr, band,
                                         bmul)
    dcs = bg.DeviceConstraintSystem(sc.cs.serialize())
    t = bg.ProverTranscript()
    gpoint, geval = bg.shift_reduction_prove(
        dcs, torch.from_numpy(sc.witness.view(np.int64)).cuda(), t,
        *((_ints(d[0]), orc.to_int(d[1]), _ints(d[2])) for d in (band, bmul)))
    assert t.finalize() == proof
    assert gpoint == _ints(point)
    assert geval == orc.to_int(out3[0])
