"""The calls a user of this library makes, as cases a program can time.

Sizes come from the benchmark and the tests: G1 MSMs from a few hundred points
(a verifier's batch) to the 2^22 points of the headline, Fr transforms up to
2^22, commits of 2^8 .. 2^16 evaluations, EIP-4844 blobs, EIP-2537 inputs and
the word-prime transform.  Device-resident calls go through the *_device entry
points on torch's current stream, host calls through the Python binding.

Every output is a whole number modulo a prime, encoded as bytes or 64-bit
words: there is one right answer, bit for bit, and no rounding.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import crypto_b200 as kb

BLS, BN = kb.CURVE_BLS12_381, kb.CURVE_BN254

# The resident SRS of the commit cases: a program loads one per process, as
# large as its largest polynomial.
SRS_LOG = 16
TAU = (0x1D3C5A7F9B2E4D6081A3C5E7F9).to_bytes(32, "little")

# Word-prime NTT: the 64-bit prime 2^64 - 2^32 + 1 with generator 7.
GOLDILOCKS, GOLDILOCKS_GEN = (1 << 64) - (1 << 32) + 1, 7


def listed():
    return [
        # A large prover's multi-exponentiation over resident points, any curve
        # points accepted: the headline.
        {"name": "msm_bls_2p22", "kind": "msm_device", "curve": BLS, "n": 1 << 22, "subgroup": False,
         "skewed": False},
        # A circuit of about a million constraints against an SRS (points known
        # to lie in G1); the size is whatever the circuit has.
        {"name": "msm_bls_g1_1000003", "kind": "msm_device", "curve": BLS, "n": 1000003, "subgroup": True,
         "skewed": False},
        # A Groth16-style witness on BN254: many zeros, ones and small values.
        {"name": "msm_bn_skewed_2p21", "kind": "msm_device", "curve": BN, "n": 1 << 21, "subgroup": False,
         "skewed": True},
        # The drop-in call on host buffers, an ordinary size.
        {"name": "msm_bls_host_100003", "kind": "msm_host", "curve": BLS, "n": 100003, "subgroup": False,
         "skewed": False},
        # The drop-in call at its smallest in earnest: a batch verifier's sum,
        # where launches and dependent latency count.
        {"name": "msm_bls_host_300", "kind": "msm_host", "curve": BLS, "n": 300, "subgroup": False,
         "skewed": False},
        # Forward transform of a large polynomial, resident.
        {"name": "ntt_bls_fwd_2p22", "kind": "ntt_device", "curve": BLS, "log_n": 22, "inverse": False,
         "coset": False, "batch": 1},
        # The quotient step of a BN254 prover: three inverse coset transforms.
        {"name": "ntt_bn_inv_coset_2p18x3", "kind": "ntt_device", "curve": BN, "log_n": 18, "inverse": True,
         "coset": True, "batch": 3},
        # One commit of 4096 evaluations against the resident SRS.
        {"name": "kzg_commit_4096", "kind": "commit", "log_n": 12},
        # An aggregator's mixed batch: uneven polynomials in one call.
        {"name": "kzg_batch_96", "kind": "batch", "count": 96, "log_lo": 8, "log_hi": 16},
        # A block builder's blob: commitment and opening proof.
        {"name": "blob_commit_and_proof", "kind": "blob", "blobs": 1},
        # The G1MSM precompile with its range, curve and subgroup checks.
        {"name": "eip2537_1000", "kind": "eip2537", "n": 1000},
        # Word-prime transform of the largest size the interface takes.
        {"name": "word_ntt_2p20", "kind": "word_ntt", "log_n": 20, "inverse": False},
    ]


def _log_uniform(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["msm_device", "msm_device", "msm_device", "msm_host", "msm_host", "ntt_device",
                       "ntt_device", "commit", "batch", "blob", "eip2537", "word_ntt"])
    if kind in ("msm_device", "msm_host"):
        n = _log_uniform(rng, 1 << 9, 1 << 22) if kind == "msm_device" else _log_uniform(rng, 64, 1 << 18)
        return {"kind": kind, "curve": rng.choice([BLS, BN]), "n": n, "subgroup": rng.random() < 0.4,
                "skewed": rng.random() < 0.3}
    if kind == "ntt_device":
        log_n = rng.randint(8, 22)
        return {"kind": kind, "curve": rng.choice([BLS, BN]), "log_n": log_n,
                "inverse": rng.random() < 0.5, "coset": rng.random() < 0.4,
                "batch": rng.randint(1, 5) if log_n <= 19 else 1}
    if kind == "commit":
        return {"kind": kind, "log_n": rng.randint(6, SRS_LOG)}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 128), "log_lo": rng.randint(6, 10),
                "log_hi": rng.randint(11, SRS_LOG)}
    if kind == "blob":
        return {"kind": kind, "blobs": rng.randint(1, 6)}
    if kind == "eip2537":
        return {"kind": kind, "n": _log_uniform(rng, 16, 1 << 16)}
    return {"kind": kind, "log_n": rng.randint(4, 20), "inverse": rng.random() < 0.5}


# ---- inputs ---------------------------------------------------------------------


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _ok(rc: int) -> None:
    if rc != 0:
        raise RuntimeError(f"call returned {rc}: {kb.last_error()}")


def _to_gpu(data: bytes) -> torch.Tensor:
    return torch.from_numpy(np.frombuffer(data, dtype=np.uint8).copy()).cuda()


def _points(curve: int, seed: int, n: int) -> torch.Tensor:
    """n points k_i * G1 with k_i uniform, wire encoding, on the GPU."""
    k = _to_gpu(kb.gen_scalars(curve, 2 * seed + 1001, n))
    pts = torch.empty(n * kb.POINT_BYTES[curve], dtype=torch.uint8, device="cuda")
    _ok(kb.lib().kb200_g1_fixed_base_device(curve, k.data_ptr(), n, pts.data_ptr(), _stream()))
    torch.cuda.current_stream().synchronize()
    return pts


def _ensure_srs() -> None:
    if kb.kzg_srs_size() != 1 << SRS_LOG:
        kb.kzg_srs_generate(TAU, 1 << SRS_LOG)


def _batch_sizes(case) -> list[int]:
    """An uneven mix of powers of two, small polynomials more frequent."""
    lo, span = case["log_lo"], case["log_hi"] - case["log_lo"] + 1
    return [1 << (lo + (i * i + 3 * i) % span * (i % 3 + 1) // 3) for i in range(case["count"])]


_blob_setup = False


def _ensure_blob_setup() -> None:
    global _blob_setup
    if not _blob_setup:
        _ok(kb.lib().kzg_blob_setup_generate(TAU))
        _blob_setup = True


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind in ("msm_device", "msm_host"):
        curve, n = case["curve"], case["n"]
        sc = kb.gen_scalars(curve, 2 * seed + 1, n, 1 if case["skewed"] else 0)
        pts = _points(curve, seed, n)
        if kind == "msm_device":
            s["scalars"], s["points"] = _to_gpu(sc), pts
            s["out"] = torch.empty(kb.POINT_BYTES[curve], dtype=torch.uint8, device="cuda")
        else:
            s["scalars"], s["points"] = sc, pts.cpu().numpy().tobytes()
    elif kind == "ntt_device":
        n = case["batch"] << case["log_n"]
        s["data"] = _to_gpu(kb.gen_scalars(case["curve"], 2 * seed + 1, n))
    elif kind == "commit":
        _ensure_srs()
        s["evals"] = kb.gen_scalars(BLS, 2 * seed + 1, 1 << case["log_n"])
    elif kind == "batch":
        _ensure_srs()
        s["sizes"] = _batch_sizes(case)
        s["evals"] = kb.gen_scalars(BLS, 2 * seed + 1, sum(s["sizes"]))
    elif kind == "blob":
        _ensure_blob_setup()
        s["data"] = []
        for b in range(case["blobs"]):
            raw = kb.gen_scalars(BLS, 64 * seed + 2 * b + 1, 4096 + 1)
            be = np.frombuffer(raw, dtype=np.uint8).reshape(-1, 32)[:, ::-1].tobytes()
            s["data"].append((be[: 4096 * 32], be[4096 * 32:]))
    elif kind == "eip2537":
        n = case["n"]
        pts = _points(BLS, seed, n).cpu().numpy().reshape(n, 2, 48)
        sc = np.frombuffer(kb.gen_scalars(BLS, 2 * seed + 1, n), dtype=np.uint8).reshape(n, 32)
        rows = np.zeros((n, 160), dtype=np.uint8)
        rows[:, 16:64] = pts[:, 0]
        rows[:, 80:128] = pts[:, 1]
        rows[:, 128:] = sc[:, ::-1]
        s["input"] = rows.tobytes()
    elif kind == "word_ntt":
        n = 1 << case["log_n"]
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        # uniform words below the modulus but for a 2^-32 sliver
        s["data"] = torch.randint(-(1 << 63), (1 << 63) - 1, (n,), dtype=torch.int64, device="cuda",
                                  generator=g)
        # up to 2^16 the root is an n-th root, above it a 2n-th root
        order = n if n <= 1 << 16 else 2 * n
        root = pow(GOLDILOCKS_GEN, (GOLDILOCKS - 1) // order, GOLDILOCKS)
        s["root"] = pow(root, -1, GOLDILOCKS) if case["inverse"] else root
        s["scratch"] = torch.empty(n, dtype=torch.int64, device="cuda")
        s["n"] = n
    return s


# ---- one pass -------------------------------------------------------------------


def run(s):
    kind, lib = s["kind"], kb.lib()
    if kind == "msm_device":
        fn = lib.kb200_msm_device_subgroup if s["subgroup"] else lib.kb200_msm_device
        _ok(fn(s["curve"], s["scalars"].data_ptr(), s["points"].data_ptr(), s["n"], s["out"].data_ptr(),
               _stream()))
        return s["out"]
    if kind == "msm_host":
        fn = kb.gpukit_multi_pippenger_subgroup if s["subgroup"] else kb.gpukit_multi_pippenger
        return np.frombuffer(fn(s["curve"], s["scalars"], s["points"], s["n"]), dtype=np.uint8)
    if kind == "ntt_device":
        _ok(lib.kb200_ntt_device(s["curve"], s["data"].data_ptr(), 1 << s["log_n"], int(s["inverse"]),
                                 int(s["coset"]), s["batch"], _stream()))
        return s["data"]
    if kind == "commit":
        return np.frombuffer(kb.kzg_commit(s["evals"]), dtype=np.uint8)
    if kind == "batch":
        return np.frombuffer(b"".join(kb.kzg_commit_batch(s["evals"], s["sizes"])), dtype=np.uint8)
    if kind == "blob":
        out = []
        for blob, z in s["data"]:
            rc, commit = kb.kzg_blob_to_commit(blob)
            _ok(rc)
            rc, proof, y = kb.kzg_commit_to_proof(blob, z)
            _ok(rc)
            out.append(np.frombuffer(commit + proof + y, dtype=np.uint8))
        return out
    if kind == "eip2537":
        rc, out = kb.bls12_381_g1_msm(s["input"])
        _ok(0 if rc == 1 else rc or -1)
        return np.frombuffer(out, dtype=np.uint8)
    _ok(lib.kb200_word_ntt_device(s["data"].data_ptr(), s["scratch"].data_ptr(), s["n"], GOLDILOCKS,
                                  s["root"], int(s["inverse"]), _stream()))
    return s["data"]


# ---- what a pass cannot do without ----------------------------------------------


def _mont(limbs: int) -> int:
    """32-bit multiply-adds of one Montgomery product, schoolbook."""
    return 4 * limbs * limbs + limbs


def _msm_madds(curve: int, n: int) -> float:
    """Bucket additions at six products each, over the best window."""
    limbs = 12 if curve == BLS else 8
    return 6 * _mont(limbs) * min(-(-256 // c) * (n + (1 << c)) for c in range(4, 17))


def work(case):
    """bytes: inputs once and outputs once; flops: two per 32-bit multiply-add."""
    kind = case["kind"]
    if kind in ("msm_device", "msm_host"):
        pb = kb.POINT_BYTES[case["curve"]]
        return {"bytes": case["n"] * (32 + pb) + pb, "flops": 2 * _msm_madds(case["curve"], case["n"])}
    if kind == "ntt_device":
        n = 1 << case["log_n"]
        return {"bytes": 64 * n * case["batch"], "flops": n * case["log_n"] * _mont(8) * case["batch"]}
    if kind in ("commit", "batch", "blob"):
        if kind == "commit":
            sizes = [1 << case["log_n"]]
        elif kind == "blob":
            sizes = [4096] * (2 * case["blobs"])
        else:
            sizes = _batch_sizes(case)
        madds = sum(_msm_madds(BLS, n) + n / 2 * math.log2(n) * _mont(8) for n in sizes)
        return {"bytes": sum(32 * n + 48 for n in sizes), "flops": 2 * madds}
    if kind == "eip2537":
        # two 64-bit doubling chains of seven products a step for the G1 check
        return {"bytes": 160 * case["n"] + 128,
                "flops": 2 * (_msm_madds(BLS, case["n"]) + case["n"] * 128 * 7 * _mont(12))}
    n = 1 << case["log_n"]
    return {"bytes": 16 * n, "flops": n * case["log_n"] * _mont(2)}


def exact(case, seed):
    """No rounding anywhere: outputs are whole numbers, compared bit for bit."""
    return None
