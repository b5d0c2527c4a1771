"""Bucket reduction by binary folding: sub-chunk sizes and windows that
exercise its edges, byte-equal to the oracle's MSM."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = r'''
import random, sys
sys.path.insert(0, "tests")
import crypto_b200 as kb, _oracle as O
from test_msm_gpu import rand_points
curve, c = %d, %d
pb = O.PB[curve]
P = {1: 0x30644e72e131a029b85045b68181585d97816a916871ca8d3c208c16d87cfd47,
     2: int("1a0111ea397fe69a4b1ba7b6434bacd764774b84f38512bf6730d2a0f6b0f6241eabfffeb153ffffb9feffffffffaaab", 16)}[curve]
def neg(pt):
    h = pb // 2
    return pt[:h] + (P - int.from_bytes(pt[h:], "big")).to_bytes(h, "big")
rng = random.Random(1000 * curve + c)
base = rand_points(curve, 64, seed=77 + c)
pt = lambda i: base[pb * (i %% 64):pb * (i %% 64 + 1)]
pts, sc = [], []
M = 1 << (c - 1)
# digits of the lowest window: neighbours of a pair hold the same point (a
# doubling in the fold), opposite points (infinity), or one is empty; the
# last bucket, the first, and both ends of sub-chunks
for k in sorted({1, 2, 3, 4, M, M - 1, M // 2, M // 2 + 1, 31, 32, 33, 255, 256, 257} & set(range(1, M + 1))):
    pts.append(pt(0)); sc.append(k)
for k in range(5, min(M, 21), 2):
    pts.append(pt(k)); sc.append(k)
    pts.append(neg(pt(k)) if k %% 4 == 1 else pt(k)); sc.append(k + 1)
for i in range(120):
    pts.append(pt(i)); sc.append(rng.randrange(O.FR[curve]))
n = len(pts)
pts = b"".join(pts)
S = b"".join(s.to_bytes(32, "little") for s in sc)
assert kb.msm_window(curve, n) == c
got = kb.gpukit_multi_pippenger(curve, S, pts, n)
assert got == O.msm(curve, S, pts, n)
print("ok")
'''


@pytest.mark.parametrize("curve", [1, 2])
@pytest.mark.parametrize("c,log_q", [(2, 5), (4, 8), (6, 5), (9, 8), (12, 6), (16, 5), (16, 8), (20, 7)])
def test_reduction_sub_chunks(cuda_lib, curve, c, log_q):
    """Windows of 2 to 2^19 buckets (one bucket block, many blocks, several
    sub-chunks per block: 2^19 at 2^7 a sub-chunk), with doublings and
    cancellations among neighbouring buckets."""
    env = dict(os.environ, KB200_MSM_RED_LOGQ=str(log_q), KB200_MSM_C=str(c), KB200_MSM_GLV_C=str(c))
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", CODE % (curve, c)], cwd=root, env=env,
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and "ok" in out.stdout, out.stdout + out.stderr


MANY = r'''
import random, sys
sys.path.insert(0, "tests")
import crypto_b200 as kb, _oracle as O
from test_msm_gpu import rand_points
curve, c, n = %d, %d, %d
pb, r = O.PB[curve], O.FR[curve]
base = rand_points(curve, 32, seed=91)
rng = random.Random(n + c)
s = [rng.randrange(r) for _ in range(n)]
tot = [sum(s[j::32]) %% r for j in range(32)]
pts = (base * (n // 32 + 1))[:pb * n]
le = lambda v: b"".join(x.to_bytes(32, "little") for x in v)
assert kb.msm_window(curve, n) == c
assert kb.gpukit_multi_pippenger(curve, le(s), pts, n) == O.msm(curve, le(tot), base, 32)
print("ok")
'''


@pytest.mark.parametrize("curve", [1, 2])
@pytest.mark.parametrize("c,n", [(6, 4001), (9, 4001), (9, 30011), (13, 30011)])
def test_buckets_over_several_chunks(cuda_lib, curve, c, n):
    """Every bucket over several accumulation chunks, some, and few of them:
    the reduction adds their further records after the load."""
    env = dict(os.environ, KB200_MSM_C=str(c), KB200_MSM_GLV_C=str(c))
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", MANY % (curve, c, n)], cwd=root, env=env,
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and "ok" in out.stdout, out.stdout + out.stderr
