"""Sign of a zero result: a float32 FMA chain whose products all underflow from
below ends in -0 in numc, also where K ends inside a slab of the kernels (the
steps past K must leave the sum as it is).  Compared by bytes."""
import numpy as np
import pytest

import numc_gb300 as nc
import oracle

from gpu_util import needs_gpu

pytestmark = [pytest.mark.gpu, needs_gpu]
torch = pytest.importorskip("torch")

PROFILES = [nc.INT8_X86_AVX2, nc.INT8_ARM_NEON]
# numc's unpacked path; every tile of the packed path's rule, K below, at and
# above multiples of the slabs (16, 32, 64) and of a 256-deep block
SHAPES = [(20, 3, 20), (33, 17, 30), (40, 96, 40), (64, 65, 64), (100, 96, 100), (300, 100, 300),
          (512, 300, 515), (33, 97, 20003), (300, 512, 1700), (1030, 270, 1100),
          (1000, 513, 1000), (1536, 100, 2100), (2000, 261, 1501), (2405, 258, 2100)]


def _operands(M, K, N, offset):
    """Products of -1e-60: below half of the smallest subnormal.  `offset`: rows
    that are not 16-byte aligned."""
    a = torch.full((M, K + offset), -1e-30, device="cuda")[:, offset:]
    b = torch.full((K, N + offset), 1e-30, device="cuda")[:, offset:]
    return a, b


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("profile", PROFILES, ids=["x86", "neon"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_gemm(shape, profile, offset):
    M, K, N = shape
    a, b = _operands(M, K, N, offset)
    out = torch.full((M, N), float("nan"), device="cuda")
    nc.gemm(a, b, out, algo=nc.ALGO_SIMT, param=profile)
    want = oracle.matmul(a.contiguous().cpu().numpy(), b.contiguous().cpu().numpy(), profile)
    assert np.signbit(want).any()
    assert out.cpu().numpy().tobytes() == want.tobytes()


def test_plan():
    probs = []
    for i, (M, K, N) in enumerate(SHAPES[:9]):
        a, b = _operands(M, K, N, i & 1)
        probs.append((a, b, torch.full((M, N), float("nan"), device="cuda")))
    plan = nc.GemmPlan(probs, nc.ALGO_SIMT)
    plan.run()
    torch.cuda.synchronize()
    for a, b, out in probs:
        want = oracle.matmul(a.contiguous().cpu().numpy(), b.contiguous().cpu().numpy())
        assert out.cpu().numpy().tobytes() == want.tobytes()
    plan.free()
