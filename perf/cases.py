"""The work that programs have this library do, as cases that can be timed.

Every case goes through the public Python entry points on one GPU.  Field
elements are BN254 Fr in Montgomery form, (n, 4) int64 tensors; every result
is an exact integer, so there is nothing here that rounds.
"""
import math
import random

import numpy as np
import torch

from provekit_b200.batch import Batch
from provekit_b200.merkle import merkle_tree, whir_commit
from provekit_b200.ntt import intt_rn, ntt_nr
from provekit_b200.poseidon2 import poseidon2_hash_many
from provekit_b200.prover import HostR1CS, prove_r1cs, whir_params_for
from provekit_b200.rs import RSFr

# Integer multiply-adds on 32-bit words that a 256-bit modular product and
# square need: 64 or 36 word products, then 64 of the reduction.
PRODUCT = 2 * (64 + 64)
SQUARE = 2 * (36 + 64)
COMPRESS = 14 * SQUARE  # a Skyscraper compression squares in 14 of its 18 rounds
FR = 32  # bytes of a field element and of a digest

TOP_LIMB = 0x30644E72E131A029  # of the modulus: limbs with a smaller top limb are reduced


def listed():
    return [
        # the smallest call of the ntt crate: NTTEngine's first table covers it, one launch
        {"name": "ntt_2p10", "kind": "ntt", "log_n": 10},
        # the inverse at the size of the single-transform benchmark
        {"name": "intt_2p16", "kind": "intt", "log_n": 16},
        # the target transform size
        {"name": "ntt_2p24", "kind": "ntt", "log_n": 24},
        # the ReedSolomon plugin with a message count, a length and masks that
        # are no powers of two (zero padding and replication inside)
        {"name": "rs_encode_12x5003", "kind": "rs", "messages": 12, "length": 5003, "masks": 60,
         "log_codeword": 15},
        # the commitment of a small circuit's last rounds: latency counts
        {"name": "commit_2p12", "kind": "commit", "log_n": 12, "folding": 3, "log_rate": 2},
        # the commitment benchmark: 2^20 coefficients, 16 messages, rate 1/4
        {"name": "commit_2p20", "kind": "commit", "log_n": 20, "folding": 4, "log_rate": 2},
        # a Merkle tree over leaves that come as bytes (the HashEngine plugin)
        {"name": "merkle_2p16x256", "kind": "merkle", "log_leaves": 16, "leaf_size": 256},
        # Poseidon2 hashes of short inputs, a count that is no power of two
        {"name": "poseidon2_200003x3", "kind": "poseidon2", "count": 200003, "length": 3},
        # uneven jobs in one graph: transform, commitment and sumcheck of each
        {"name": "batch_12", "kind": "batch", "jobs": 12, "low": 10, "high": 18, "pick": 1},
        # whole proofs: the smallest served size, a ragged one with public
        # inputs, and the headline
        {"name": "prove_2p14", "kind": "prove", "constraints": 1 << 14, "inputs": 1 << 12,
         "public": 0},
        {"name": "prove_300007", "kind": "prove", "constraints": 300007, "inputs": 75001,
         "public": 5},
        {"name": "prove_2p20", "kind": "prove", "constraints": 1 << 20, "inputs": 1 << 18,
         "public": 0},
    ]


def _between(rng, low, high):
    """A whole number spread over the logarithm of [low, high]."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["ntt", "intt", "rs", "commit", "merkle", "poseidon2", "batch", "prove",
                       "prove"])
    if kind == "ntt":
        # columns: interleaved transforms over the same points
        log_n = rng.randint(10, 22)
        return {"kind": kind, "log_n": log_n,
                "columns": rng.randint(1, 12) if log_n <= 18 else rng.randint(1, 3)}
    if kind == "intt":
        return {"kind": kind, "log_n": rng.randint(10, 22)}
    if kind == "rs":
        length = _between(rng, 100, 60000)
        messages = rng.randint(1, 17)
        return {"kind": kind, "messages": messages, "length": length,
                "masks": rng.choice([0, rng.randint(1, 10 * messages)]),
                "log_codeword": (length - 1).bit_length() + rng.randint(1, 3)}
    if kind == "commit":
        return {"kind": kind, "log_n": rng.randint(12, 20), "folding": rng.randint(1, 5),
                "log_rate": rng.randint(1, 3)}
    if kind == "merkle":
        return {"kind": kind, "log_leaves": rng.randint(4, 18),
                "leaf_size": 32 * rng.randint(1, 24)}
    if kind == "poseidon2":
        return {"kind": kind, "count": _between(rng, 100, 400000), "length": rng.randint(1, 7)}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(3, 14), "low": 10, "high": rng.randint(12, 18),
                "pick": rng.randint(2, 1 << 20)}
    constraints = _between(rng, 1 << 14, 1 << 20)
    return {"kind": kind, "constraints": constraints, "inputs": max(16, constraints // 4),
            "public": rng.choice([0, 0, rng.randint(1, 12)])}


def _fr(count, seed):
    """count reduced field elements on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    v = torch.empty((count, 4), dtype=torch.int64, device="cuda")
    v[:, :3] = torch.randint(-(1 << 63), (1 << 63) - 1, (count, 3), generator=g,
                             dtype=torch.int64, device="cuda")
    v[:, 3] = torch.randint(0, TOP_LIMB, (count,), generator=g, dtype=torch.int64, device="cuda")
    return v


def _log_sizes(case):
    rng = random.Random(case["pick"])
    return [rng.randint(case["low"], case["high"]) for _ in range(case["jobs"])]


class _Memory:
    """Memory that a batch owns, for torch.as_tensor."""

    def __init__(self, address, shape, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (address, False), "shape": shape,
                                         "typestr": typestr, "version": 3}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("ntt", "intt"):
        n = 1 << case["log_n"]
        return {"kind": kind, "n": n, "values": _fr(n * case.get("columns", 1), seed)}
    if kind == "rs":
        M, L = case["messages"], case["length"]
        return {"kind": kind, "rs": RSFr(), "messages": _fr(M * L, seed).reshape(M, L, 4),
                "masks": _fr(case["masks"], seed + 1) if case["masks"] else None,
                "codeword": 1 << case["log_codeword"]}
    if kind == "commit":
        return {"kind": kind, "coeffs": _fr(1 << case["log_n"], seed),
                "folding": case["folding"], "log_rate": case["log_rate"]}
    if kind == "merkle":
        size = case["leaf_size"]
        leaves = _fr((size << case["log_leaves"]) // FR, seed).view(torch.uint8).reshape(-1)
        return {"kind": kind, "leaves": leaves, "leaf_size": size}
    if kind == "poseidon2":
        return {"kind": kind, "inputs": _fr(case["count"] * case["length"], seed),
                "length": case["length"]}
    if kind == "batch":
        batch = Batch(_log_sizes(case), seed)
        outputs = []
        for j in range(case["jobs"]):
            job = batch.job(j)
            rows = job.num_leaves
            # 2^3 messages at rate 1/4: a codeword of 4n field elements
            for address, shape, typestr in ((job.ntt, (job.n, 4), "<i8"),
                                            (job.codeword, (4 * job.n, 4), "<i8"),
                                            (job.layers, (FR * (2 * rows - 1),), "|u1")):
                outputs.append(torch.as_tensor(_Memory(address, shape, typestr, batch),
                                               device="cuda"))
        return {"kind": kind, "batch": batch, "outputs": outputs, "jobs": case["jobs"],
                "stream": torch.cuda.Stream()}
    host = HostR1CS(seed, case["constraints"], case["inputs"], case["public"])
    return {"kind": kind, "r1cs": host.to_device(), "whir": whir_params_for(host),
            "blinding_seed": seed + 1}


def run(state):
    kind = state["kind"]
    if kind == "ntt":
        return ntt_nr(state["values"], state["n"], 1)
    if kind == "intt":
        return intt_rn(state["values"])
    if kind == "rs":
        return state["rs"].interleaved_encode(state["messages"], state["masks"],
                                              state["codeword"])
    if kind == "commit":
        return whir_commit(state["coeffs"], state["folding"], state["log_rate"])
    if kind == "merkle":
        return merkle_tree(state["leaves"], state["leaf_size"])
    if kind == "poseidon2":
        return poseidon2_hash_many(state["inputs"], state["length"])
    if kind == "batch":
        # graphs are captured on a stream of their own; its results are read
        # on the host, so a program waits for it
        state["batch"].run(stream=state["stream"])
        state["stream"].synchronize()
        sumchecks = []
        for j in range(state["jobs"]):
            got = state["batch"].sumcheck_result(j)
            sumchecks.append(np.concatenate([got[k].reshape(-1) for k in
                                             ("r", "coeffs", "alpha", "rho", "sum_g",
                                              "blinding_eval")]))
        return state["outputs"], np.concatenate(sumchecks)
    fields, commitment, proof = prove_r1cs(state["r1cs"], state["whir"],
                                           blinding_seed=state["blinding_seed"])
    fields["root"] = np.frombuffer(fields["root"], np.uint8)
    fields["transcript"] = np.array(fields["transcript"], np.uint64)
    return fields, commitment, proof


def _ntt_products(n, columns=1, skipped=0):
    return columns * n // 2 * (n.bit_length() - 1 - skipped)


def _commit_work(n, folding, log_rate):
    """(bytes, operations) of encoding n coefficients and hashing the rows."""
    rows = (n >> folding) << log_rate
    row = 1 << folding
    work = _ntt_products(rows, row, log_rate) * PRODUCT
    work += rows * (row - 1) * COMPRESS + (rows - 1) * COMPRESS
    return FR * (n + rows * row + 2 * rows - 1), work


def work(case):
    kind = case["kind"]
    if kind in ("ntt", "intt"):
        n, columns = 1 << case["log_n"], case.get("columns", 1)
        return {"bytes": 2 * FR * n * columns, "flops": _ntt_products(n, columns) * PRODUCT}
    if kind == "rs":
        M, rows = case["messages"], 1 << case["log_codeword"]
        coset = 1 << max(0, case["length"] + case["masks"] // M - 1).bit_length()
        skipped = max(0, case["log_codeword"] - (coset.bit_length() - 1))
        return {"bytes": FR * (M * case["length"] + case["masks"] + M * rows),
                "flops": _ntt_products(rows, M, skipped) * PRODUCT}
    if kind == "commit":
        b, f = _commit_work(1 << case["log_n"], case["folding"], case["log_rate"])
        return {"bytes": b, "flops": f}
    if kind == "merkle":
        n, size = 1 << case["log_leaves"], case["leaf_size"]
        return {"bytes": n * size + FR * (2 * n - 1),
                "flops": (n * (size // FR - 1) + n - 1) * COMPRESS}
    if kind == "poseidon2":
        n, length = case["count"], case["length"]
        permutations = n * max(1, -(-length // 3))
        # 8 full rounds of 4 sboxes, 56 partial ones of one and four diagonal products
        each = (8 * 4 + 56) * (2 * SQUARE + PRODUCT) + 56 * 4 * PRODUCT
        return {"bytes": FR * n * (length + 1), "flops": permutations * each}
    if kind == "batch":
        b = f = 0
        for log_n in _log_sizes(case):
            n = 1 << log_n
            cb, cf = _commit_work(n, 3, 2)
            b += cb + FR * 6 * n
            f += cf + _ntt_products(n) * PRODUCT + 14 * n * PRODUCT
        return {"bytes": b, "flops": f}
    # the witness and its blinding polynomial committed together, the zk
    # sumcheck over four tables, then rounds that commit an eighth each time
    nc, nw = case["constraints"], 1 + case["inputs"] + case["constraints"]
    m = max(13, (nw - 1).bit_length())
    b, f = _commit_work(1 << (m + 1), 4, 2)
    k = m - 3
    while k >= 6:
        cb, cf = _commit_work(1 << k, 3, 2)
        b, f, k = b + cb, f + cf, k - 3
    b += FR * (nw + 5 * nc)
    f += (14 * nc + 6 * nw + 9 * (1 << m)) * PRODUCT
    return {"bytes": b, "flops": f}
