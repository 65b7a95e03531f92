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


@pytest.mark.parametrize("profile", PROFILES, ids=["x86", "neon"])
@pytest.mark.parametrize("shape", [(20, 3, 20), (47, 45, 50), (130, 33, 130), (300, 100, 300),
                                   (257, 300, 515), (1000, 513, 1000), (2100, 259, 1900)],
                         ids=lambda s: "x".join(map(str, s)))
def test_float64(shape, profile):
    M, K, N = shape
    a, b = np.full((M, K), -1e-200), np.full((K, N), 1e-200)
    out = torch.full((M, N), float("nan"), dtype=torch.float64, device="cuda")
    nc.gemm(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), out, algo=nc.ALGO_SIMT,
            param=profile)
    want = oracle.matmul(a, b, profile)
    assert np.signbit(want).any()
    assert out.cpu().numpy().tobytes() == want.tobytes()


@pytest.mark.parametrize("dt,tiny", [("float32", 1e-30), ("float64", 1e-200)])
def test_naive(dt, tiny):
    """numc_matmul_naive: products rounded to -0 and added to +0."""
    M, K, N = 70, 45, 90
    a, b = np.full((M, K), -tiny, dt), np.full((K, N), tiny, dt)
    with nc.Ctx() as ctx:
        A, B, C = ctx.from_numpy(a), ctx.from_numpy(b), ctx.zeros((M, N), dt)
        nc.matmul_naive(A, B, C)
        assert C.numpy().tobytes() == oracle.matmul(a, b, oracle.PROFILE_WRAP).tobytes()


@pytest.mark.parametrize("K", [37, 300])
def test_strides_beyond_32_bits(K):
    """Strides that the float32 tiles' offsets do not hold: the general kernel."""
    M, N, wide = 3, 20000, 1 << 24
    a = torch.full((M, wide), -1e-30, device="cuda")[:, :K]
    b = torch.full((K, N), 1e-30, device="cuda")
    out = torch.full((M, N), float("nan"), device="cuda")
    nc.gemm(a, b, out, algo=nc.ALGO_SIMT, param=nc.INT8_X86_AVX2)
    want = oracle.matmul(a.contiguous().cpu().numpy(), b.cpu().numpy())
    assert np.signbit(want).any()
    assert out.cpu().numpy().tobytes() == want.tobytes()
