"""Grouped plans where the persistent kernels change over: more tiles per block
than one look-up of 32 covers, and tiles deeper than the accumulator buffers,
next to tiles of a single slab."""
import numpy as np
import pytest

import numc_gb300 as nc
import oracle
from numc_gb300 import synth

from gpu_util import needs_gpu, rel_err_vs_scale

pytestmark = [pytest.mark.gpu, needs_gpu]
torch = pytest.importorskip("torch")


def f16_bound(K):   # two float16 planes, three products, float32 sums
    return 4 * 2.0 ** -22 + 2 * (3 * K + 2) * 2.0 ** -24


def operands(M, N, K, seed):
    a, b = synth.operands("uniform", M, K, N, dtype="float32", seed=seed)
    return a, b, torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()


@pytest.mark.parametrize("param,N", [(64, 72 * 64 - 3), (128, 72 * 128 - 5)])
def test_many_tiles_per_block(param, N):
    dims = [(72 * 128 - 7, N, 40), (200, 300, 1500), (129, 65, 641), (1, 1, 3000), (300, 200, 64)]
    probs = []
    for i, (M, n, K) in enumerate(dims):
        a, b, ta, tb = operands(M, n, K, 50 + i)
        out = torch.full((M, n), float("nan"), device="cuda")
        probs.append((a, b, ta, tb, out))
    plan = nc.GemmPlan([(p[2], p[3], p[4]) for p in probs], nc.ALGO_SPLIT_FP16, param)
    plan.run()
    nc.check_status()
    for a, b, _, _, out in probs:
        M, K = a.shape
        rows = np.unique(np.linspace(0, M - 1, 200).astype(int))
        got = out.cpu().numpy()
        assert np.isfinite(got).all()
        assert rel_err_vs_scale(got[rows], oracle.matmul(a[rows], b), a[rows], b) <= f16_bound(K)
    plan.free()
