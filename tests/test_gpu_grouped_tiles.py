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


def simt_dims(which):
    if which == "one":       # alone: the small tiles
        return [(33, 65, 300)]
    if which == "unpacked":  # numc's unpacked path, 16 x 16 and 32 x 32 tiles
        return [(m, n, k) for m in (1, 15, 33) for n in (1, 31, 50) for k in (1, 64, 70)] * 40
    # enough work that 128 x 64 tiles are worth it, with every kind of remainder
    return [(m, n, k) for m in (127, 128, 131, 520) for n in (63, 64, 67, 500)
            for k in (60, 255, 256, 257, 600)] + [(3, 7, 0), (2000, 1900, 17), (5000, 5000, 16)]


@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("which", ["one", "unpacked", "many"])
def test_cuda_core_tiles_are_the_single_kernels(which, transposed):
    gen = torch.Generator(device="cuda").manual_seed(5)
    probs = []
    for M, N, K in simt_dims(which):
        a = torch.randn((K, M) if transposed else (M, K), device="cuda", generator=gen)
        b = torch.randn((N, K) if transposed else (K, N), device="cuda", generator=gen)
        out = torch.full((M, N), float("nan"), device="cuda")
        probs.append((a.t(), b.t(), out) if transposed else (a, b, out))
    plan = nc.GemmPlan(probs, nc.ALGO_SIMT)
    plan.run(graph=True)
    nc.check_status()
    for a, b, out in probs:
        want = torch.empty_like(out)
        nc.gemm(a, b, want, algo=nc.ALGO_SIMT)
        assert torch.equal(out, want), (a.shape, b.shape)
    plan.free()


def test_strides_beyond_32_bit_offsets():
    # 3 rows 20 million elements apart: the general tile
    wide = torch.zeros(2 * 20_000_000 + 400, device="cuda")
    a = wide.as_strided((3, 400), (20_000_000, 1))
    a.copy_(torch.randn(3, 400, device="cuda"))
    b = torch.randn(400, 1000, device="cuda")
    out, want = torch.empty(3, 1000, device="cuda"), torch.empty(3, 1000, device="cuda")
    plan = nc.GemmPlan([(a, b, out)], nc.ALGO_SIMT)
    plan.run()
    nc.gemm(a, b, want, algo=nc.ALGO_SIMT)
    nc.check_status()
    assert torch.equal(out, want)
