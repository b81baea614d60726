"""Device entry points recorded into CUDA graphs: those that return with work queued on their stream can
be captured once a call of their kind has run (a fold even before), at sizes on either side of the
lines between their kernels, and a replay computes on what the buffers then hold."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA device", allow_module_level=True)

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = """
import ctypes
import numpy as np, torch
import oracle as orc
import binius64_b200 as bg
from binius64_b200 import constraint_system as csm, eval_form as ef
from binius64_b200._ffi import check, lib

def replayed(f, fill, seeds=(1, 2)):
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    fill(0)
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        f()
    for seed in seeds:
        fill(seed)
        g.replay()
        torch.cuda.synchronize()
        yield seed

def filler(buf):
    def fill(seed):
        buf.copy_(bg.to_device(orc.random_elems(np.random.default_rng(seed), len(buf))))
    return fill

def merkle(name, elems, log_leaves, log_batch, nodes):
    check(getattr(lib(), name)(elems.data_ptr(), log_leaves, log_batch, nodes.data_ptr(),
                               torch.cuda.current_stream().cuda_stream))
"""

TREES = PRELUDE + """
# the only tree before the capture is one of other kernels
for entry, ref, warm in (("binius_merkle_commit", orc.merkle_commit, 14),
                         ("binius_merkle_commit_vision4", orc.vision4_merkle_commit, WARM_V4)):
    big = torch.empty(((2 << warm) - 1, 32), dtype=torch.uint8, device="cuda")
    merkle(entry, torch.zeros((1 << warm, 2), dtype=torch.int64, device="cuda"), warm, 0, big)
    torch.cuda.synchronize()
    for log_leaves, log_batch in ((4, 2), (9, 0)) if WARM_V4 > 12 else ((13, 0),):
        elems = torch.empty((1 << (log_leaves + log_batch), 2), dtype=torch.int64, device="cuda")
        nodes = torch.empty(((2 << log_leaves) - 1, 32), dtype=torch.uint8, device="cuda")
        for seed in replayed(lambda: merkle(entry, elems, log_leaves, log_batch, nodes),
                             filler(elems)):
            want = ref(bg.to_host(elems), log_leaves, log_batch).reshape(-1, 32)
            assert np.array_equal(nodes.cpu().numpy(), want), (entry, log_leaves, seed)
print("ok")
"""

OTHERS = PRELUDE + """
for d, se, sl in ((8, 0, 0), (11, 1, 0), (12, 0, 3), (17, 2, 1)):
    ntt, tw = bg.AdditiveNTT(d), orc.domain_twiddles(d)
    data = torch.empty((1 << d, 2), dtype=torch.int64, device="cuda")
    ntt.forward_transform(data, se, sl)
    for seed in replayed(lambda: ntt.forward_transform(data, se, sl), filler(data)):
        src = orc.random_elems(np.random.default_rng(seed), 1 << d)
        assert np.array_equal(bg.to_host(data), orc.ntt_forward(tw, d, src, se, sl)), (d, seed)

for log_len, b in ((5, 3), (9, 4)):
    ch = [orc.to_int(x) for x in orc.random_elems(np.random.default_rng(b), b)]
    cw = torch.empty((1 << (log_len + b), 2), dtype=torch.int64, device="cuda")
    out = bg.empty_elems(1 << log_len)
    bg.fold_interleaved(cw, ch, log_len, b, out=out)
    for seed in replayed(lambda: bg.fold_interleaved(cw, ch, log_len, b, out=out), filler(cw)):
        want = orc.fri_fold_interleaved(bg.to_host(cw), log_len, b,
                                        np.array([orc.from_int(c) for c in ch], dtype=np.uint64))
        assert np.array_equal(bg.to_host(out), want), (log_len, seed)

for log_len, k in ((8, 2), (18, 4)):
    ch = [orc.to_int(x) for x in orc.random_elems(np.random.default_rng(k), k)]
    ntt, tw = bg.AdditiveNTT(log_len), orc.domain_twiddles(log_len)
    cw = torch.empty((1 << log_len, 2), dtype=torch.int64, device="cuda")
    out = bg.empty_elems(1 << (log_len - k))
    bg.fold_codeword(ntt, cw, ch, log_len, out=out)
    for seed in replayed(lambda: bg.fold_codeword(ntt, cw, ch, log_len, out=out), filler(cw)):
        want = orc.fri_fold_codeword(tw, log_len, bg.to_host(cw), log_len,
                                     np.array([orc.from_int(c) for c in ch], dtype=np.uint64))
        assert np.array_equal(bg.to_host(out), want), (log_len, seed)

circ = csm.synthetic_circuit(10, 900, 4, seed=3)
code, n_values = ef.synthetic_program(circ)
prog, batch = ef.EvalForm(code, n_values), 3
n_in = circ.cs.layout.committed_total_len - circ.cs.layout.n_internal
v = torch.zeros((n_values, batch), dtype=torch.int64, device="cuda")
plain = torch.empty_like(v)
def fill(seed):
    torch.manual_seed(seed)
    v.zero_()
    v[:n_in] = torch.randint(-2**62, 2**62, (n_in, batch), dtype=torch.int64, device="cuda")
    plain.copy_(v)
prog.evaluate(plain.view(-1), batch)
for seed in replayed(lambda: prog.evaluate(v.view(-1), batch), fill):
    prog.evaluate(plain.view(-1), batch)
    assert torch.equal(v, plain), seed
print("ok")
"""

FIRST = PRELUDE + """
# nothing of the library has run: a fold needs no handle that was made before
log_len, b = 8, 3
ch = [orc.to_int(x) for x in orc.random_elems(np.random.default_rng(b), b)]
cw = torch.empty((1 << (log_len + b), 2), dtype=torch.int64, device="cuda")
out = bg.empty_elems(1 << log_len)
for seed in replayed(lambda: bg.fold_interleaved(cw, ch, log_len, b, out=out), filler(cw)):
    want = orc.fri_fold_interleaved(bg.to_host(cw), log_len, b,
                                    np.array([orc.from_int(c) for c in ch], dtype=np.uint64))
    assert np.array_equal(bg.to_host(out), want), seed
print("ok")
"""


@pytest.mark.parametrize("script", [TREES.replace("WARM_V4", "13"), TREES.replace("WARM_V4", "6"),
                                    OTHERS, FIRST],
                         ids=["small trees after large", "large trees after small", "others",
                              "first call"])
def test_captured(script):
    out = subprocess.run([sys.executable, "-c", script], cwd=ROOT, capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0 and out.stdout.strip().endswith("ok"), out.stdout + out.stderr
