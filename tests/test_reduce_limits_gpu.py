"""Bucket reduction at its limits: windows of 2^20 and 2^21 buckets, which have the
most blocks, sub-chunks and points a block leaves, and fold without groups; and
sub-chunk sizes forced against the planner's at many points."""
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
curve, c, n = %d, %d, %d
r = O.FR[curve]
base = rand_points(curve, 32, seed=91)
rng = random.Random(n + c)
# windows whose lowest digits are the first and last buckets, then random ones
M = 1 << (c - 1) if c else 1 << 15
s = ([1, 2, M, M - 1, M // 2, M // 2 + 1, r - 1, r - M] + [rng.randrange(r) for _ in range(n)])[:n]
tot = [sum(s[j::32]) %% r for j in range(32)]
le = lambda v: b"".join(x.to_bytes(32, "little") for x in v)
pts = (base * (n // 32 + 1))[:O.PB[curve] * n]
want = O.msm(curve, le(tot), base, 32)
if c:
    assert kb.msm_window(curve, n) == c
assert kb.gpukit_multi_pippenger(curve, le(s), pts, n) == want
assert kb.gpukit_multi_pippenger_subgroup(curve, le(s), pts, n) == want
print("ok")
'''


@pytest.mark.parametrize("curve", [1, 2])
@pytest.mark.parametrize("c,n,log_q", [(21, 4000, 5), (21, 4000, 8), (22, 4000, 5), (22, 4000, 8),
                                       (0, 1 << 17, 5), (0, 1 << 17, 8), (0, 1 << 20, 5), (0, 1 << 20, 8)])
def test_reduction_limits(cuda_lib, curve, c, n, log_q):
    env = dict(os.environ, KB200_MSM_RED_LOGQ=str(log_q))
    if c:
        env.update(KB200_MSM_C=str(c), KB200_MSM_GLV_C=str(c))
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", CODE % (curve, c, n)], cwd=root, env=env,
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and "ok" in out.stdout, out.stdout + out.stderr
