"""
The work a user has this framework do, as timed cases: BN254 G1 MSMs, Fr NTTs,
batches of both, whole Groth16-shaped jobs, element-wise field and point
arithmetic and the 64-bit-field NTT, each through its public entry point.

Sizes are those of the benchmark's configurations (NTT 2^10..2^24, MSM 2^10..2^22,
jobs of 2^12..2^20, 64-bit NTT 2^16..2^24) and odd ones between them. A case is a
dict of a `kind` and that kind's sizes and options. Inputs are made from the seed
on the device or by zkgpu.workloads; every output is whole numbers (limbs of
canonical field elements, affine coordinates), the same for any correct program.
"""

from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "zk-gpu-accelerator_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from zkgpu import batch, curve_gpu, msm_gpu, ntt_gpu, prover, workloads as wl  # noqa: E402
from zkgpu.field256_gpu import BN254_FQ, BN254_FR  # noqa: E402

# a prime below 2^31 with 2-adicity 23, and one of 63 bits with 2-adicity 32
_P31 = 998244353
_P63 = (2**31 - 7) * 2**32 + 1
_COSET = 5


def listed() -> list[dict]:
    return [
        # the smallest MSM a caller sends to the GPU: latency and launches
        {"name": "msm_1000", "kind": "msm", "n": 1000, "scalars": "uniform"},
        # the plain single-instance MSM configuration
        {"name": "msm_2e16", "kind": "msm", "n": 1 << 16, "scalars": "uniform"},
        # a witness commitment: skewed scalars, a size that is no power of two
        {"name": "msm_witness_777777", "kind": "msm", "n": 777_777, "scalars": "skewed"},
        # the largest MSM, the headline
        {"name": "msm_2e22", "kind": "msm", "n": 1 << 22, "scalars": "uniform"},
        # the smallest NTT configuration, forward
        {"name": "ntt_2e12", "kind": "ntt", "log_n": 12, "invert": False, "coset": False},
        # the middle NTT configuration, inverse (evaluations to coefficients)
        {"name": "intt_2e20", "kind": "ntt", "log_n": 20, "invert": True, "coset": False},
        # the largest NTT with the coset option, the headline (low-degree extension)
        {"name": "coset_ntt_2e24", "kind": "ntt", "log_n": 24, "invert": False, "coset": True},
        # a batch of transforms of uneven sizes in one launch
        {"name": "ntt_batch_24", "kind": "ntt_batch", "log_min": 10, "log_max": 18, "jobs": 24},
        # a service's MSMs of uneven sizes over its resident base set's table
        {"name": "msm_table_8", "kind": "msm_table", "log_base": 17, "log_min": 12, "jobs": 8},
        # one proof from its host inputs: 7 transforms and 4 MSMs
        {"name": "proof_2e14", "kind": "proof", "log_n": 14},
        # element-wise point arithmetic (mixed additions of a commitment vector), ragged
        {"name": "g1_add_affine_300001", "kind": "g1", "op": "add_affine", "n": 300_001},
        # the 64-bit field's transform
        {"name": "ntt64_2e22", "kind": "ntt64", "log_n": 22, "mod": _P63, "invert": False},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    """An integer spread over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng) -> dict:
    kind = rng.choice(["msm", "msm", "ntt", "ntt", "ntt_batch", "msm_table", "proof", "g1", "field", "ntt64"])
    if kind == "msm":
        return {"kind": kind, "n": _log_int(rng, 1000, 1 << 22), "scalars": rng.choice(["uniform", "skewed"])}
    if kind == "ntt":
        return {"kind": kind, "log_n": rng.randint(10, 24), "invert": rng.random() < 0.5, "coset": rng.random() < 0.5}
    if kind == "ntt_batch":
        return {"kind": kind, "log_min": 10, "log_max": rng.randint(12, 19), "jobs": rng.randint(2, 64)}
    if kind == "msm_table":
        return {"kind": kind, "log_base": rng.randint(13, 19), "log_min": 12, "jobs": rng.randint(1, 24)}
    if kind == "proof":
        return {"kind": kind, "log_n": rng.randint(12, 18)}
    if kind == "g1":
        return {"kind": kind, "op": rng.choice(["add", "add_affine", "double"]), "n": _log_int(rng, 1000, 1 << 20)}
    if kind == "field":
        return {"kind": kind, "op": rng.choice(["mul", "add"]), "field": rng.choice(["fr", "fq"]),
                "n": _log_int(rng, 1000, 1 << 23)}
    return {"kind": kind, "log_n": rng.randint(16, 23), "mod": rng.choice([_P31, _P63]), "invert": rng.random() < 0.5}


# ---- inputs -----------------------------------------------------------------


def _rows(seed: int, n: int) -> torch.Tensor:
    """(n, 4) uint64 device rows uniform below 2^253, so canonical in both fields."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.randint(-(2**63), 2**63 - 1, (n, 4), dtype=torch.int64, device="cuda", generator=g)
    r[:, 3] &= (1 << 61) - 1
    return r.view(torch.uint64)


def _scalars(case: dict, seed: int, n: int) -> torch.Tensor:
    make = wl.skewed_scalars if case.get("scalars") == "skewed" else wl.uniform_fr
    return torch.from_numpy(make(seed, n)).cuda()


def _points(seed: int, n: int) -> torch.Tensor:
    """(n, 2, 4) affine rows of points k_i G of the whole group."""
    return curve_gpu.mul_generator(_rows(seed, n))


def _sizes(case: dict, seed: int, top: int) -> list[int]:
    """The sizes of a batch's jobs, log-uniform up to 2^top; the same for every seed."""
    rng = np.random.default_rng(case["jobs"] * 64 + top)
    return [int(2**v) for v in rng.uniform(case["log_min"], top, size=case["jobs"])]


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    st: dict = {"case": case}
    if kind == "msm":
        st["points"], st["scalars"] = _points(seed, case["n"]), _scalars(case, seed + 1, case["n"])
    elif kind == "ntt":
        st["x"] = _rows(seed, 1 << case["log_n"])
    elif kind == "ntt_batch":
        logs = [int(math.log2(n)) for n in _sizes(case, seed, case["log_max"] + 1)]
        st["xs"] = [_rows(seed + k, 1 << min(e, case["log_max"])) for k, e in enumerate(logs)]
        # a prover's mix: a third each of inverse, coset and inverse coset transforms
        st["invert"] = [k % 3 != 1 for k in range(case["jobs"])]
        st["coset"] = [None if k % 3 == 0 else _COSET for k in range(case["jobs"])]
    elif kind == "msm_table":
        st["table"] = msm_gpu.FixedBaseTable(_points(seed, 1 << case["log_base"]), 16)
        st["scalars"] = [torch.from_numpy((wl.skewed_scalars if k % 4 else wl.uniform_fr)(seed + k, n)).cuda()
                         for k, n in enumerate(_sizes(case, seed, case["log_base"]))]
    elif kind == "proof":
        m = 1 << case["log_n"]
        bases = _points(seed, m)
        st["table"] = msm_gpu.FixedBaseTable(bases, 16)
        st["job"] = prover.ProofJob(prover.synthetic_request(seed + 1, m), bases)
        st["workspaces"] = {}
    elif kind == "g1":
        n = case["n"]
        one = BN254_FQ.from_ints([1]).reshape(1, 1, 4).expand(n, 1, 4)
        # Jacobian points with Z != 1: doubles of affine ones
        st["a"] = curve_gpu.double(torch.cat([_points(seed, n), one], dim=1))
        if case["op"] == "add":
            st["b"] = curve_gpu.double(torch.cat([_points(seed + 1, n), one], dim=1))
        elif case["op"] == "add_affine":
            st["b"] = _points(seed + 1, n)
    elif kind == "field":
        st["a"], st["b"] = _rows(seed, case["n"]), _rows(seed + 1, case["n"])
        st["field"] = BN254_FR if case["field"] == "fr" else BN254_FQ
    else:
        g = torch.Generator(device="cuda").manual_seed(seed)
        st["x"] = torch.randint(0, case["mod"], (1 << case["log_n"],), dtype=torch.int64, device="cuda", generator=g)
    return st


# ---- one pass ---------------------------------------------------------------


def _coords(points) -> np.ndarray:
    """The affine coordinates of host Points as 64-bit limbs, x then y (zeros for the identity)."""
    out = np.zeros((len(points), 8), dtype=np.uint64)
    for row, p in zip(out, points):
        if not p.is_identity():
            x, y = p.affine()
            row[:] = np.frombuffer(x.to_bytes(32, "little") + y.to_bytes(32, "little"), dtype=np.uint64)
    return out


def run(st: dict):
    out = _call(st)
    # the same 64 bits as signed words, which torch also indexes
    if isinstance(out, list):
        return [t.view(torch.int64) for t in out]
    return out.view(torch.int64) if isinstance(out, torch.Tensor) else out


def _call(st: dict):
    case = st["case"]
    kind = case["kind"]
    if kind == "msm":
        return _coords([msm_gpu.msm_pippenger_rows(st["points"], st["scalars"])])
    if kind == "ntt":
        return BN254_FR.ntt(st["x"], invert=case["invert"], coset=_COSET if case["coset"] else None)
    if kind == "ntt_batch":
        return batch.ntt_batch(st["xs"], invert=st["invert"], coset=st["coset"])
    if kind == "msm_table":
        return _coords(batch.msm_fixed_batch(st["table"], st["scalars"]))
    if kind == "proof":
        job = st["job"]
        prover.prove_plain(job, st["workspaces"], table=st["table"])
        return {"h": job.h_plain, "msms": _coords(list(job.msm_points().values()))}
    if kind == "g1":
        if case["op"] == "double":
            return curve_gpu.double(st["a"])
        return (curve_gpu.add if case["op"] == "add" else curve_gpu.add_affine)(st["a"], st["b"])
    if kind == "field":
        return (st["field"].mul if case["op"] == "mul" else st["field"].add)(st["a"], st["b"])
    return ntt_gpu.ntt_gpu(st["x"], case["mod"], case["invert"])


def exact(case: dict, seed: int):
    """Every output is whole numbers, equal or wrong: there is nothing to approximate in 64 bits."""
    return None


# ---- the work of a pass -------------------------------------------------------

# 32-bit multiply-adds of one 256-bit Montgomery product (8 x 8 words, twice, and 8), two operations each
_PRODUCT = 2 * 136


def _msm_work(n: int) -> tuple[float, float]:
    """Points and scalars read once; a mixed addition (10 products) per point and 16-bit window of 254 bits."""
    return 96.0 * n, 16.0 * n * 10 * _PRODUCT


def _ntt_work(log_n: int, coset: bool = False) -> tuple[float, float]:
    n = 1 << log_n
    return 64.0 * n, (n / 2 * log_n + (n if coset else 0)) * _PRODUCT


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "msm":
        b, f = _msm_work(case["n"])
    elif kind == "ntt":
        b, f = _ntt_work(case["log_n"], case["coset"])
    elif kind == "ntt_batch":
        logs = [min(int(math.log2(n)), case["log_max"]) for n in _sizes(case, 0, case["log_max"] + 1)]
        parts = [_ntt_work(e, k % 3 != 0) for k, e in enumerate(logs)]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif kind == "msm_table":
        parts = [_msm_work(n) for n in _sizes(case, 0, case["log_base"])]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif kind == "proof":
        parts = [_ntt_work(case["log_n"], k >= 3) for k in range(7)] + [_msm_work(1 << case["log_n"])] * 4
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif kind == "g1":
        products, rows = {"add": (16, 9), "add_affine": (11, 8), "double": (7, 6)}[case["op"]]
        b, f = 32.0 * rows * case["n"], products * _PRODUCT * case["n"]
    elif kind == "field":
        b, f = 96.0 * case["n"], (_PRODUCT if case["op"] == "mul" else 16) * case["n"]
    else:
        # a 64-bit product reduced by a precomputed quotient: three 64-bit multiplies of four 32-bit ones
        n = 1 << case["log_n"]
        b, f = 16.0 * n, n / 2 * case["log_n"] * 24
    return {"bytes": b, "flops": f}
