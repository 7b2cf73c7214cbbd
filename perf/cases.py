"""What this framework is timed on: the calls a Groth16 prover over BN254 makes, by size.

A case is one call through the public Python mirror of the C ABI.  Its `kind`
says which:

  prove   CudaCircuit.prove_with_blinders: a witness in host memory in, a proof out
  batch   CudaBackend.prove_batch: many proofs over several keys in one submission
  msm     CudaMsm.msm_g1 / msm_g2 (host buffers) or the _device forms
  ntt     CudaNtt (host buffers) or ntt_device, in all five modes

The key of a circuit and the bases of an MSM are fixed for a size, as a
deployment's are; the witness, the blinders, the scalars and the transformed
values come from the seed.  Everything is exact arithmetic on whole numbers, so
every output is compared byte for byte (and there is no rounding for a 64-bit
reference to measure).
"""
import functools
import math
import random

import numpy as np
import torch

import snarkrs_b200 as S

N_INPUTS, N_PUBLIC = 256, 16          # as bench.py's circuits
MSM_MAX = {1: 1 << 20, 2: 1 << 18}    # the largest standalone MSM of each group here

# 8 circuits, log-uniform over 2^12 .. 2^18 constraints (bench.py's batched workload)
BATCH_SIZES = "4326,5379,11019,19079,39385,50483,55274,133345"


def listed():
    return [
        # a small circuit (a hash or a signature check): latency, launches and
        # the bucket reduction's serial depth decide
        {"name": "prove-500", "kind": "prove", "constraints": 500},
        # an ordinary circuit, domain 2^16 (sha256 of a short message, a Merkle path)
        {"name": "prove-2e15", "kind": "prove", "constraints": 1 << 15},
        # the headline: an identity-credential circuit, 1.1M constraints, domain 2^21
        {"name": "prove-1.1M", "kind": "prove", "constraints": 1100000},
        # a proving service's submission: 64 proofs over 8 keys of uneven size
        {"name": "batch-64", "kind": "batch", "sizes": BATCH_SIZES, "each": 8},
        # a small commitment opened from host buffers
        {"name": "msm-g1-1000-host", "kind": "msm", "group": 1, "n": 1000, "dist": 0, "form": 0, "where": "host"},
        # a polynomial commitment: uniform scalars, bases resident
        {"name": "msm-g1-2e20", "kind": "msm", "group": 1, "n": 1 << 20, "dist": 0, "form": 0, "where": "device"},
        # a witness commitment: 70% zeros and ones, Montgomery form, ragged length
        {"name": "msm-g1-300007-sparse", "kind": "msm", "group": 1, "n": 300007, "dist": 1, "form": 1,
         "where": "device"},
        # the G2 half of a commitment key
        {"name": "msm-g2-2e18", "kind": "msm", "group": 2, "n": 1 << 18, "dist": 0, "form": 0, "where": "device"},
        # a mid-size transform in device memory
        {"name": "ntt-forward-2e16", "kind": "ntt", "mode": "forward", "log_n": 16, "where": "device"},
        # the prover's chain at a large size, in device memory
        {"name": "ntt-chain-2e22", "kind": "ntt", "mode": "intt-coset-ntt", "log_n": 22, "where": "device"},
        # a small inverse coset transform on a host buffer with the caller's shift
        {"name": "ntt-coset-inv-2e12-host", "kind": "ntt", "mode": "coset-inverse", "log_n": 12, "where": "host"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("prove", "prove", "batch", "msm", "msm", "msm", "ntt", "ntt", "ntt"))
    if kind == "prove":
        return {"kind": kind, "constraints": _log_uniform(rng, 300, 600000)}
    if kind == "batch":
        sizes = sorted(_log_uniform(rng, 1 << 9, 1 << 17) for _ in range(rng.randint(2, 5)))
        return {"kind": "batch", "sizes": ",".join(map(str, sizes)), "each": rng.randint(2, 8)}
    where = rng.choice(("device", "device", "host"))
    if kind == "msm":
        group = rng.choice((1, 1, 2))
        return {"kind": "msm", "group": group, "n": _log_uniform(rng, 1, MSM_MAX[group]), "dist": rng.randint(0, 1),
                "form": rng.randint(0, 1), "where": where}
    modes = ("forward", "inverse", "intt-coset-ntt", "coset-forward", "coset-inverse")
    return {"kind": "ntt", "mode": rng.choice(modes), "log_n": rng.randint(1, 18 if where == "host" else 22),
            "where": where}


MODES = {"forward": S.NTT_FORWARD, "inverse": S.NTT_INVERSE, "intt-coset-ntt": S.NTT_INTT_COSET_NTT,
         "coset-forward": S.NTT_COSET_FORWARD, "coset-inverse": S.NTT_COSET_INVERSE}


@functools.lru_cache(maxsize=None)
def _backend():
    return S.CudaBackend(0)


@functools.lru_cache(maxsize=16)
def _circuit(constraints):
    """The key of this size, prepared on the GPU, and its witness generator."""
    synth = S.SynthCircuit(7000 + constraints, constraints, N_INPUTS, N_PUBLIC)
    key = S.ProvingKey.from_bytes(synth.zkey(11, device=0), check_points=False)
    return synth, _backend().prepare(key)


@functools.lru_cache(maxsize=2)
def _points(group):
    return S.synth_points(group, 77, MSM_MAX[group])


@functools.lru_cache(maxsize=2)
def _points_on_gpu(group):
    return torch.frombuffer(bytearray(_points(group)), dtype=torch.uint8).cuda()


def _fr(rng):
    return S.fr_to_mont_bytes(rng.randrange(1, S.R_MOD))


def _elements(n, seed):
    """n uniform values below 2^253 (canonical whatever the modulus), as 8 words each."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randint(-(1 << 31), 1 << 31, (n, 8), dtype=torch.int64, device="cuda", generator=gen)
    x[:, 7] &= (1 << 29) - 1
    return x.to(torch.int32)


def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    if kind == "prove":
        synth, circuit = _circuit(case["constraints"])
        return {"kind": kind, "circuit": circuit, "witness": synth.witness(seed), "r": _fr(rng), "s": _fr(rng)}
    if kind == "batch":
        jobs = []
        for size in case["sizes"].split(","):
            synth, circuit = _circuit(int(size))
            jobs += [(circuit, synth.witness(seed * 64 + j), _fr(rng), _fr(rng)) for j in range(case["each"])]
        rng.shuffle(jobs)
        return {"kind": kind, "backend": _backend(), "jobs": jobs}
    if kind == "msm":
        group, n = case["group"], case["n"]
        scalars = S.synth_scalars(seed, n, case["dist"])
        if case["form"]:   # a prover's own vector: Montgomery form
            scalars = _to_montgomery(scalars)
        state = {"kind": kind, "msm": S.CudaMsm(_backend()), "group": group, "n": n, "form": case["form"],
                 "where": case["where"]}
        if case["where"] == "host":
            return {**state, "bases": _points(group)[:n * (64 if group == 1 else 128)], "scalars": scalars}
        return {**state, "bases": _points_on_gpu(group),
                "scalars": torch.frombuffer(bytearray(scalars), dtype=torch.uint8).cuda()}
    state = {"kind": kind, "ntt": S.CudaNtt(_backend()), "mode": case["mode"], "log_n": case["log_n"],
             "where": case["where"], "shift": _fr(rng) if case["mode"].startswith("coset") else None}
    data = _elements(1 << case["log_n"], seed)
    return {**state, "data": data.cpu().numpy().tobytes() if case["where"] == "host" else data}


@functools.lru_cache(maxsize=1)
def _montgomery_cache():
    return {0: bytes(32), 1: S.fr_to_mont_bytes(1)}


def _to_montgomery(scalars):
    small = _montgomery_cache()
    out = []
    for i in range(0, len(scalars), 32):
        v = int.from_bytes(scalars[i:i + 32], "little")
        out.append(small[v] if v < 2 else ((v << 256) % S.R_MOD).to_bytes(32, "little"))
    return b"".join(out)


def _bytes(raw):
    return np.frombuffer(raw, dtype=np.uint8)


def run(state):
    kind = state["kind"]
    if kind == "prove":
        return _bytes(state["circuit"].prove_with_blinders(state["witness"], state["r"], state["s"]).to_bytes())
    if kind == "batch":
        return _bytes(b"".join(p.to_bytes() for p in state["backend"].prove_batch(state["jobs"])))
    if kind == "msm":
        msm, g2 = state["msm"], state["group"] == 2
        if state["where"] == "host":
            fn = msm.msm_g2 if g2 else msm.msm_g1
            return _bytes(fn(state["bases"], state["scalars"], state["form"]))
        fn = msm.msm_g2_device if g2 else msm.msm_g1_device
        return _bytes(fn(state["bases"].data_ptr(), state["scalars"].data_ptr(), state["n"], state["form"]))
    ntt, mode, shift = state["ntt"], state["mode"], state["shift"]
    if state["where"] == "device":   # in place
        ntt.ntt_device(MODES[mode], state["log_n"], state["data"].data_ptr(), shift)
        return state["data"]
    if mode == "intt-coset-ntt":
        return _bytes(ntt.intt_coset_ntt(state["data"]))
    if mode.startswith("coset"):
        return _bytes(ntt.coset_ntt(state["data"], shift, inverse=mode == "coset-inverse"))
    return _bytes(ntt.ntt(state["data"], inverse=mode == "inverse"))


# ---- work: whole-number operations, a 32 x 32 -> 64-bit multiply-add counted as two ----
PRODUCT = 2 * (2 * 8 * 8 + 8)                 # one Montgomery product of 8 words
ADD = {1: 6 * PRODUCT, 2: 3 * 6 * PRODUCT}    # one affine addition, its inversion shared (Fq2: three Fq products)


def _msm_work(group, n, terms):
    """terms scalars that reach the buckets: one addition per window at the width that makes
    windows times (terms + buckets) smallest."""
    adds = min(-(-255 // c) * (terms + 2 ** c) for c in range(4, 23))
    return {"bytes": n * (32 + 64 * group) + 64 * group, "flops": adds * ADD[group]}


def _chain_work(n, vectors):
    """iNTT, coset multiply, NTT of each vector."""
    return vectors * n * (math.log2(n) + 1) * PRODUCT


def _prove_work(constraints):
    wires = constraints + N_INPUTS + 1
    n = 1 << (constraints + N_PUBLIC).bit_length()
    # 60% of a witness is 0 or 1, 20% below 2^32: about a quarter of the windows are used
    parts = [_msm_work(1, wires, wires * 0.25) for _ in range(3)] + [_msm_work(2, wires, wires * 0.25),
                                                                     _msm_work(1, n, n)]
    return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts) + _chain_work(n, 3)}


def work(case):
    kind = case["kind"]
    if kind == "prove":
        return _prove_work(case["constraints"])
    if kind == "batch":
        each = [_prove_work(int(s)) for s in case["sizes"].split(",")]
        return {k: case["each"] * sum(w[k] for w in each) for k in ("bytes", "flops")}
    if kind == "msm":
        n = case["n"]
        return _msm_work(case["group"], n, n if case["dist"] == 0 else max(1, 0.3 * n))
    n = 1 << case["log_n"]
    chain = 2 if case["mode"] == "intt-coset-ntt" else 1
    return {"bytes": 64 * n, "flops": (chain * n / 2 * case["log_n"] + (n if "coset" in case["mode"] else 0)) * PRODUCT}


def tolerance(case):
    return "exact"
