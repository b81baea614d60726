"""A wait for the tensor cores that runs out (one that nothing completes, of a few polls) reaches the
caller: the status query, reads of results, the calls that wait and the calls that would launch such
work all return the timeout status.  The report stands for the rest of a process, so each run is a
process of its own; no wait here leaves work on the GPU."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA device", allow_module_level=True)

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import numpy as np, torch
import binius64_b200 as bg
from binius64_b200 import _ffi
from binius64_b200 import constraint_system as csm

T = _ffi.BINIUS_E_TIMEOUT
L = _ffi.lib()

def code(f):
    try:
        f()
    except _ffi.BiniusError as e:
        return e.code
    return 0

circ = csm.synthetic_circuit(10, 800, 1, seed=1)
cs = bg.DeviceConstraintSystem(circ.cs.serialize())
prover = bg.Prover(cs, 1)
words = torch.from_numpy(circ.witness.view(np.int64)).cuda()
ntt = bg.AdditiveNTT(11)
data = torch.zeros((1 << 11, 2), dtype=torch.int64, device="cuda")
small, wide = bg.AdditiveNTT(5), bg.AdditiveNTT(12)
calls = {
    "transform": lambda: ntt.forward_transform(data),
    "inverse": lambda: ntt.inverse_transform(data),
    "encode": lambda: bg.ReedSolomonCode(11, 1).encode_batch(wide, data, 0),
    "fold": lambda: bg.fold_interleaved(data, [3, 5], 9, 2),
    "prove": lambda: prover.prove(words),
    "prove_host": lambda: prover.prove_host(circ.witness),
    "tree": lambda: bg.BinaryMerkleTreeProver().commit(data, 2),
    "read": lambda: bg.to_host(data),
    "status": bg.device_status,
}
assert {k: code(f) for k, f in calls.items()} == dict.fromkeys(calls, 0)
if WITH_GRAPH:
    # the wait as a graph's node: reported by the replay, not by the capture
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        _ffi.check(L.binius_debug_tensor_wait(torch.cuda.current_stream().cuda_stream))
    assert code(calls["status"]) == 0
    g.replay()
else:
    _ffi.check(L.binius_debug_tensor_wait(None))
torch.cuda.synchronize()
small.forward_transform(data[:1 << 5])  # waits for nothing
got = {k: code(f) for k, f in calls.items()}
assert got == dict.fromkeys(calls, T), got
assert b"tensor" in L.binius_last_error()
torch.cuda.synchronize()  # the context itself is sound
assert int((data + 1).sum().item()) == data.numel()
print("ok")
"""


@pytest.mark.parametrize("with_graph", [False, True])
def test_wait_that_runs_out_is_reported(with_graph):
    out = subprocess.run([sys.executable, "-c", f"WITH_GRAPH = {with_graph}\n" + SCRIPT], cwd=ROOT,
                         capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip().endswith("ok"), out.stdout + out.stderr
