"""float32 on the CUDA cores with packed FMAs: bit-identical to numc's packed
path (the oracle's AVX2 and NEON profiles) on every tile size of its rule,
ragged last tiles, remainder register tiles and K-block ends included."""
import numpy as np
import pytest

import numc_gb300 as nc
import oracle
from numc_gb300 import synth

from gpu_util import needs_gpu

pytestmark = [pytest.mark.gpu, needs_gpu]
torch = pytest.importorskip("torch")

# one or more problems per tile (32 x 32, 32 x 64, 64 x 64, 128 x 64, 128 x 80,
# 128 x 96), K around the 16-deep slabs and 256-deep blocks
SHAPES = [(512, 300, 515), (33, 17, 20003), (9001, 257, 40), (300, 512, 1700), (700, 31, 650),
          (1030, 270, 1100), (1000, 513, 1000), (1536, 100, 2100), (2000, 261, 1501),
          (2048, 40, 2048), (2405, 258, 2100), (3000, 300, 2501)]


def _run(a, b, profile, out=None, bias=None):
    if out is None:
        out = torch.full((a.shape[0], b.shape[1]), float("nan"), device="cuda")
    nc.gemm(a, b, out, algo=nc.ALGO_SIMT, param=profile)
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("profile", [nc.INT8_X86_AVX2, nc.INT8_ARM_NEON], ids=["x86", "neon"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_bit_identical_to_numc(shape, profile):
    M, K, N = shape
    a, b = synth.operands("uniform", M, K, N, seed=3)
    got = _run(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), profile)
    want = oracle.matmul(a, b, profile)
    assert got.tobytes() == want.tobytes()


@pytest.mark.parametrize("form", ["a_transposed", "b_transposed", "both", "strided", "offset",
                                  "out_transposed"])
def test_strides(form):
    M, K, N = 1003, 530, 1130
    a, b = synth.operands("uniform", M, K, N, seed=4)
    ta, tb, out = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), None
    if form in ("a_transposed", "both"):
        ta = ta.t().contiguous().t()
    if form in ("b_transposed", "both"):
        tb = tb.t().contiguous().t()
    if form == "strided":
        w = torch.zeros((2 * M, 3 * K), device="cuda")
        w[::2, ::3] = ta
        ta = w[::2, ::3]
        w = torch.zeros((K, 2 * N), device="cuda")
        w[:, ::2] = tb
        tb = w[:, ::2]
    if form == "offset":
        w = torch.zeros((M, K + 1), device="cuda")
        w[:, 1:] = ta
        ta = w[:, 1:]
        out = torch.zeros((M, N + 1), device="cuda")[:, 1:]
    if form == "out_transposed":
        out = torch.zeros((N, M), device="cuda").t()
    got = _run(ta, tb, nc.INT8_ARM_NEON, out)
    assert got.tobytes() == oracle.matmul(a, b, nc.INT8_ARM_NEON).tobytes()


def test_linear_bias_and_special_values():
    M, K, N = 1000, 600, 1001
    a, b = synth.operands("normal", M, K, N, seed=5)
    a[7, 3], a[999, 599], b[2, 1000], b[11, 4] = np.inf, np.nan, -np.inf, 1e-42
    bias = synth.array("uniform", (N,), seed=5, stream=9)
    nc.set_algo("float32", nc.ALGO_SIMT, nc.INT8_ARM_NEON)
    try:
        with nc.Ctx() as ctx:
            C = ctx.zeros((M, N), "float32")
            nc.linear(ctx.from_numpy(a), ctx.from_numpy(b), ctx.from_numpy(bias), C)
            got = C.numpy()
    finally:
        nc.set_algo("float32", nc.ALGO_SIMT)
    with np.errstate(invalid="ignore"):
        want = oracle.matmul(a, b, nc.INT8_ARM_NEON) + bias
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert got[ok].tobytes() == want[ok].tobytes()


# small tiles (16 x 16 and 32 x 32, packed and unpacked path): tile edges, K
# around the slabs of 32 and 64, operands that 16-byte copies take and others
SMALL = [(1, 1, 1), (16, 64, 16), (17, 65, 15), (96, 96, 96), (95, 97, 96), (10, 1000, 80),
         (256, 128, 10), (64, 256, 64), (64, 257, 64), (100, 1024, 33), (256, 784, 128),
         (130, 600, 260), (512, 300, 512), (511, 301, 513), (2, 3000, 1000)]


@pytest.mark.parametrize("profile", [nc.INT8_X86_AVX2, nc.INT8_ARM_NEON], ids=["x86", "neon"])
@pytest.mark.parametrize("shape", SMALL, ids=lambda s: "x".join(map(str, s)))
def test_small_tiles_bit_identical(shape, profile):
    M, K, N = shape
    a, b = synth.operands("uniform", M, K, N, seed=6)
    want = oracle.matmul(a, b, profile).tobytes()
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    at, bt = ta.t().contiguous().t(), tb.t().contiguous().t()
    wide = torch.zeros((M, K + 1), device="cuda")
    wide[:, 1:] = ta
    for x, y in ((ta, tb), (at, bt), (ta, bt), (wide[:, 1:], tb)):
        assert _run(x, y, profile).tobytes() == want
