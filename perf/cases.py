"""The work whose time is followed: what a program that proves, commits, folds and generates
witnesses with this package calls, over the range of sizes that it is used at.

Kinds of case (`kind` of a case dict):

* ``prove``: a whole proof of a constraint system (`Prover.prove` over a device witness, or
  `Prover.prove_host` over host words), SHA-256 or Vision-4 Merkle trees.
* ``queue``: several proofs of uneven sizes through `ProveQueue`, as a server runs them.
* ``commit``: `commit_interleaved` of a message (Reed-Solomon encode, Merkle tree), followed by
  FRI folds of the codeword.
* ``ntt``: one additive NTT or its inverse in place, with skipped layers.
* ``sumcheck``: a bivariate product sumcheck driven round by round from the host.
* ``witness``: a circuit's witness words computed from its inputs for a batch of instances.

All results are integers or bytes: field elements, digests, proofs, words.
"""
from __future__ import annotations

import numpy as np
import torch

import binius64_b200 as bg
from binius64_b200 import constraint_system as csm
from binius64_b200 import eval_form as ef


def _n_and(log_words: int) -> int:
    """The AND constraints of a circuit that fills its words as the bench's circuits do."""
    return (1 << log_words) - (1 << (log_words - 4))


def _prove(name, log_words, n_mul, log_inv_rate=1, host=False, merkle="sha256", n_and=None):
    n_and = _n_and(log_words) - 2 * n_mul if n_and is None else n_and
    return {"name": name, "kind": "prove", "log_words": log_words, "n_and": n_and,
            "n_mul": n_mul, "log_inv_rate": log_inv_rate, "host": host, "merkle": merkle}


def _commit(name, log_len, log_inv_rate, log_batch, folds):
    return {"name": name, "kind": "commit", "log_len": log_len, "log_inv_rate": log_inv_rate,
            "log_batch": log_batch, "folds": folds}


def listed():
    return [
        # the smallest statements of the batched mix: a proof is a chain of short launches
        _prove("prove_2p12", 12, 4),
        # a hash preimage circuit of a few KiB, proved once from host words
        _prove("prove_host_2p16", 16, 1, host=True),
        # a multiplication-heavy statement at the lower code rate, its constraint count ragged
        _prove("prove_mul_2p18_rate2", 18, 256, log_inv_rate=2, n_and=201_337),
        # the headline statement: a hash preimage circuit of 64 KiB
        _prove("prove_2p20", 20, 1),
        # a proof meant for recursion: Vision-4 trees
        _prove("prove_vision4_2p14", 14, 16, merkle="vision4"),
        # a server's mix of small and middle statements, proved side by side
        {"name": "queue_mix", "kind": "queue", "log_words": "12,13,14,14,15,16,17,12",
         "workers": 8},
        # the witness commitment of a large statement, with the first FRI fold rounds
        _commit("commit_2p20_x16_folds", 20, 1, 4, 3),
        # one polynomial at the lower rate: no interleaving, leaves of one element
        _commit("commit_2p22_x1_rate2", 22, 2, 0, 2),
        # a wide interleaved trace: 64 columns, the largest commitment
        _commit("commit_2p20_x64", 20, 1, 6, 0),
        # interpolation of evaluations, some layers skipped on either side
        {"name": "intt_2p20", "kind": "ntt", "log_len": 20, "skip_early": 1, "skip_late": 2,
         "inverse": True},
        # a protocol that drives its own sumcheck over device multilinears
        {"name": "sumcheck_2p20", "kind": "sumcheck", "n_vars": 20},
        # witnesses of a batch of requests for one circuit
        {"name": "witness_2p13_x32", "kind": "witness", "log_words": 13, "batch": 32},
    ]


def draw(rng):
    kind = rng.choice(["prove", "prove", "queue", "commit", "commit", "ntt", "sumcheck",
                       "witness"])
    if kind == "prove":
        merkle = "vision4" if rng.random() < 0.15 else "sha256"
        lw = rng.randint(11, 14) if merkle == "vision4" else rng.randint(11, 20)
        n_mul = int(2 ** rng.uniform(0, max(0.0, min(lw, 18) - 10)))
        n_and = int(2 ** rng.uniform(lw - 1.5, lw - 0.1)) - 2 * n_mul
        c = _prove("", lw, n_mul, log_inv_rate=rng.choice([1, 1, 2]) if lw < 20 else 1,
                   host=rng.random() < 0.3, merkle=merkle, n_and=n_and)
        del c["name"]
        return c
    if kind == "queue":
        sizes = [rng.randint(12, 17) for _ in range(rng.randint(3, 8))]
        return {"kind": "queue", "log_words": ",".join(map(str, sizes)),
                "workers": rng.choice([4, 8, 16])}
    if kind == "commit":
        log_inv_rate, log_batch = rng.randint(1, 2), rng.randint(0, 6)
        log_len = rng.randint(12, min(24, 25 - log_batch))
        c = _commit("", log_len, log_inv_rate, log_batch, rng.randint(0, 2))
        del c["name"]
        return c
    if kind == "ntt":
        log_len = rng.randint(8, 23)
        return {"kind": "ntt", "log_len": log_len, "skip_early": rng.randint(0, 3),
                "skip_late": rng.randint(0, 4), "inverse": rng.random() < 0.6}
    if kind == "sumcheck":
        return {"kind": "sumcheck", "n_vars": rng.randint(6, 22)}
    return {"kind": "witness", "log_words": rng.randint(10, 13), "batch": rng.randint(1, 64)}


# -------------------------------------------------------------------------------- preparation

def _statement(log_words, n_and, n_mul, log_inv_rate, merkle, seed):
    circ = csm.synthetic_circuit(log_words, n_and, n_mul, seed=seed)
    cs = bg.DeviceConstraintSystem(circ.cs.serialize())
    return bg.Prover(cs, log_inv_rate, merkle_hash=merkle), circ.witness


def _elems(n, gen):
    return torch.randint(-2**63, 2**63 - 1, (n, 2), dtype=torch.int64, device="cuda",
                         generator=gen)


def _ints(rng, n):
    return [int(a) | (int(b) << 64)
            for a, b in rng.integers(0, 2**64, size=(n, 2), dtype=np.uint64)]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "prove":
        s["prover"], w = _statement(case["log_words"], case["n_and"], case["n_mul"],
                                    case["log_inv_rate"], case["merkle"], seed)
        s["host"] = case["host"]
        s["witness"] = w if case["host"] else torch.from_numpy(w.view(np.int64)).cuda()
    elif kind == "queue":
        s["queue"] = bg.ProveQueue(case["workers"])
        s["statements"] = []
        for i, lw in enumerate(int(x) for x in case["log_words"].split(",")):
            n_mul = 1 << (lw - 10)
            p, w = _statement(lw, _n_and(lw) - 2 * n_mul, n_mul, 1, "sha256", 64 * seed + i)
            s["statements"].append((p, torch.from_numpy(w.view(np.int64)).cuda()))
        torch.cuda.synchronize()
    elif kind == "commit":
        log_len, rate, b = case["log_len"], case["log_inv_rate"], case["log_batch"]
        basis = bg.standard_domain_rs_basis(log_len + b, b)
        s["ntt"] = bg.AdditiveNTT(log_len, basis=basis)
        s["params"] = bg.FRIParams(bg.ReedSolomonCode(log_len - rate, rate), b, [], 0)
        s["merkle"] = bg.BinaryMerkleTreeProver()
        s["message"] = _elems(1 << (log_len - rate + b), gen)
        s["challenges"] = [_ints(rng, b if i == 0 and b else 4) for i in range(case["folds"])]
    elif kind == "ntt":
        s["case"] = case
        s["ntt"] = bg.AdditiveNTT(case["log_len"])
        s["input"] = _elems(1 << case["log_len"], gen)
        s["data"] = torch.empty_like(s["input"])
    elif kind == "sumcheck":
        n = case["n_vars"]
        s["inputs"] = (_elems(1 << n, gen), _elems(1 << n, gen))
        s["work"] = tuple(torch.empty_like(t) for t in s["inputs"])
        s["sum"], s["challenges"] = _ints(rng, 1)[0], _ints(rng, n)
    else:
        lw = case["log_words"]
        circ = csm.synthetic_circuit(lw, _n_and(lw) - 8, 4, seed=lw)  # one circuit a size
        code, n_values = ef.synthetic_program(circ)
        s["program"], s["batch"] = ef.EvalForm(code, n_values), case["batch"]
        n_in = circ.cs.layout.committed_total_len - circ.cs.layout.n_internal
        v = torch.zeros((n_values, case["batch"]), dtype=torch.int64, device="cuda")
        v[:n_in] = torch.randint(-2**63, 2**63 - 1, (n_in, case["batch"]), dtype=torch.int64,
                                 device="cuda", generator=gen)
        s["values"] = v.view(-1)
    return s


# ---------------------------------------------------------------------------------- one pass

def _bytes(b):
    return np.frombuffer(b, dtype=np.uint8)


def run(state):
    kind = state["kind"]
    if kind == "prove":
        if state["host"]:
            return _bytes(state["prover"].prove_host(state["witness"]))
        return _bytes(state["prover"].prove(state["witness"]).finalize())
    if kind == "queue":
        q = state["queue"]
        tickets = [q.submit(p, w) for p, w in state["statements"]]
        return [_bytes(q.wait(t)[0]) for t in tickets]
    if kind == "commit":
        params = state["params"]
        out = bg.commit_interleaved(params, state["ntt"], state["merkle"], state["message"])
        outs = [out.codeword, out.committed.nodes, _bytes(out.commitment)]
        cur, n = out.codeword, params.rs_code.log_len()
        for i, ch in enumerate(state["challenges"]):
            if i == 0 and params.log_batch_size:
                cur = bg.fold_interleaved(cur, ch, n, params.log_batch_size)
            else:
                cur = bg.fold_codeword(state["ntt"], cur, ch, n)
                n -= len(ch)
            outs.append(cur)
        return outs
    if kind == "ntt":
        c, data = state["case"], state["data"]
        data.copy_(state["input"])  # the caller keeps its evaluations
        f = state["ntt"].inverse_transform if c["inverse"] else state["ntt"].forward_transform
        f(data, c["skip_early"], c["skip_late"])
        return data
    if kind == "sumcheck":
        for dst, src in zip(state["work"], state["inputs"]):
            dst.copy_(src)  # the prover folds its multilinears in place
        p = bg.BivariateProductSumcheckProver(*state["work"], state["sum"])
        vals = []
        for r in state["challenges"]:
            vals += p.execute()
            p.fold(r)
        vals += p.finish()
        return _bytes(b"".join(v.to_bytes(16, "little") for v in vals))
    fails, first = state["program"].evaluate(state["values"], state["batch"])
    return [state["values"], fails, first]


# ------------------------------------------------------------------------- what a pass needs

def _prove_bytes(log_words, n_and, n_mul):
    # the witness words, and each operand term once (a u32 word index, a shift, a constraint);
    # the synthetic circuits have six terms per AND and per MUL on average
    return 8 * (1 << log_words) + 10 * 6 * (n_and + n_mul)


def work(case):
    kind = case["kind"]
    if kind == "prove":
        n = _prove_bytes(case["log_words"], case["n_and"], case["n_mul"])
    elif kind == "queue":
        n = sum(_prove_bytes(lw, _n_and(lw), 1 << (lw - 10))
                for lw in (int(x) for x in case["log_words"].split(",")))
    elif kind == "commit":
        log_len, b = case["log_len"], case["log_batch"]
        elems = (1 << (log_len - case["log_inv_rate"] + b)) + (1 << (log_len + b))
        cur = log_len + b
        for i in range(case["folds"]):
            cur -= b if i == 0 and b else 4
            elems += 1 << cur
        n = 16 * elems + 32 * ((2 << log_len) - 1)
    elif kind == "ntt":
        n = 2 * 16 << case["log_len"]
    elif kind == "sumcheck":
        n = 2 * 16 << case["n_vars"]
    else:
        # a read of every input word and a write of every computed one
        n = 8 * case["batch"] * (1 << case["log_words"])
    return {"bytes": n, "flops": 0}


def exact(case, seed):
    """Every output is a whole number or a string of bytes."""
    return None
