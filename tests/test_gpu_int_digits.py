"""16-, 32- and 64-bit integers as digit products on the tensor cores: every
result equals the oracle's wrapped sum and the CUDA-core kernel's, bit for bit
(integers: no tolerance)."""
import numpy as np
import pytest

import numc_gb300 as nc
import oracle

from gpu_util import needs_gpu

pytestmark = [pytest.mark.gpu, needs_gpu]
torch = pytest.importorskip("torch")

DTYPES = ["int16", "uint16", "int32", "uint32", "int64", "uint64"]
# tiles of 128 x 64 / 128, K steps of 16, stages of 16 to 64, accumulation
# chains of 512, 256 and 128, K splits of short and long problems
SHAPES = [(512, 512, 512), (129, 2049, 65), (128, 2048, 128), (1000, 100, 1000),
          (513, 1111, 321), (1, 9001, 1), (3, 6000, 2), (640, 527, 1030)]


def _rand(dt, shape, seed):
    info = np.iinfo(dt)
    rng = np.random.default_rng(seed)
    return rng.integers(info.min, info.max, shape, dtype=dt, endpoint=True)


def _dev(x):
    """A CUDA tensor of x's bytes (torch has no full set of unsigned types)."""
    return torch.from_numpy(x.view(x.dtype.name.replace("uint", "int"))).cuda()


def _gemm(dt, ta, tb, out, algo, ws):
    rc = nc.lib().numc_cuda_gemm(
        nc.CODE[dt], algo, -1, ta.data_ptr(), tb.data_ptr(), out.data_ptr(), ta.shape[0],
        ta.shape[1], tb.shape[1], ta.stride(0), ta.stride(1), tb.stride(0), tb.stride(1),
        out.stride(0), out.stride(1), ws.data_ptr() if ws is not None else None,
        ws.numel() if ws is not None else 0, torch.cuda.current_stream().cuda_stream)
    nc.check(rc)
    nc.check_status()
    return out.cpu().numpy().view(dt)


def _both(dt, ta, tb, out_like):
    """(tensor-core result, CUDA-core result)."""
    M, K, N = ta.shape[0], ta.shape[1], tb.shape[1]
    need = nc.workspace_size(dt, nc.ALGO_DEFAULT, -1, M, K, N)
    assert need > 0, "this problem does not take the tensor cores"
    ws = torch.full((need,), 0x5A, dtype=torch.uint8, device="cuda")
    tc = _gemm(dt, ta, tb, out_like(), nc.ALGO_DEFAULT, ws)
    simt = _gemm(dt, ta, tb, out_like(), nc.ALGO_SIMT, None)
    return tc, simt


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("dt", DTYPES)
def test_equals_oracle_and_cuda_cores(dt, shape):
    M, K, N = shape
    a, b = _rand(dt, (M, K), 1), _rand(dt, (K, N), 2)
    ta, tb = _dev(a), _dev(b)
    tc, simt = _both(dt, ta, tb, lambda: torch.full((M, N), 77, dtype=ta.dtype, device="cuda"))
    np.testing.assert_array_equal(tc, oracle.matmul(a, b))
    np.testing.assert_array_equal(tc, simt)


@pytest.mark.parametrize("dt", DTYPES)
def test_extreme_digits(dt):
    """Every digit -128: the sums of a chain reach 2^24 exactly and leave the
    range of the fast conversion; and every digit 127."""
    bits = 8 * np.dtype(dt).itemsize
    for v in (sum(0x80 << 8 * i for i in range(bits // 8)), sum(0x7F << 8 * i for i in range(bits // 8))):
        x = (-v if v >> (bits - 1) & 1 else v) % (1 << bits)
        a = np.full((256, 1030), x, dtype=f"uint{bits}").view(dt)
        b = np.full((1030, 512), x, dtype=f"uint{bits}").view(dt)
        ta, tb = _dev(a), _dev(b)
        tc, _ = _both(dt, ta, tb, lambda: torch.zeros((256, 512), dtype=ta.dtype, device="cuda"))
        np.testing.assert_array_equal(tc, oracle.matmul(a, b))


@pytest.mark.parametrize("dt", ["int16", "int32", "int64"])
@pytest.mark.parametrize("form", ["transposed", "strided", "offset", "broadcast", "out_columns"])
def test_strides_and_alignment(dt, form):
    M, K, N = 300, 700, 520
    a, b = _rand(dt, (M, K), 3), _rand(dt, (K, N), 4)
    ta, tb = _dev(a), _dev(b)
    out = lambda: torch.zeros((M, N), dtype=ta.dtype, device="cuda")  # noqa: E731
    if form == "transposed":
        ta, tb = ta.t().contiguous().t(), tb.t().contiguous().t()
    elif form == "strided":
        wa = torch.zeros((2 * M, 3 * K), dtype=ta.dtype, device="cuda")
        wa[::2, ::3] = ta
        ta = wa[::2, ::3]
    elif form == "offset":   # rows that are not 16-byte aligned
        wa = torch.zeros((M, K + 3), dtype=ta.dtype, device="cuda")
        wa[:, 1:K + 1] = ta
        ta = wa[:, 1:K + 1]
        wide = torch.zeros((M, N + 1), dtype=ta.dtype, device="cuda")
        out = lambda: wide.zero_()[:, 1:]  # noqa: E731
    elif form == "broadcast":
        a = np.broadcast_to(a[:1], (M, K))
        ta = ta[:1].expand(M, K)
    else:                    # out column-major
        out = lambda: torch.zeros((N, M), dtype=ta.dtype, device="cuda").t()  # noqa: E731
    tc, simt = _both(dt, ta, tb, out)
    np.testing.assert_array_equal(tc, oracle.matmul(np.ascontiguousarray(a), b))
    np.testing.assert_array_equal(tc, simt)


def test_without_a_workspace_and_under_capture():
    """No workspace, or too little: the CUDA cores, as before.  With one the
    call can be captured."""
    M, K, N = 512, 640, 512
    a, b = _rand("int32", (M, K), 5), _rand("int32", (K, N), 6)
    ta, tb = _dev(a), _dev(b)
    want = oracle.matmul(a, b)
    out = torch.zeros((M, N), dtype=torch.int32, device="cuda")
    small = torch.zeros(256, dtype=torch.uint8, device="cuda")
    for ws in (None, small):
        np.testing.assert_array_equal(_gemm("int32", ta, tb, out.zero_(), nc.ALGO_DEFAULT, ws), want)
    ws = torch.zeros(nc.workspace_size("int32", nc.ALGO_DEFAULT, -1, M, K, N),
                     dtype=torch.uint8, device="cuda")
    nc.gemm(ta, tb, out, workspace=ws)
    torch.cuda.synchronize()
    out.zero_()
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        nc.gemm(ta, tb, out, workspace=ws, stream=s)
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("dt", ["int16", "uint32", "int64"])
@pytest.mark.parametrize("resident", [False, True])
def test_numc_arrays_linear_and_bmm(dt, resident):
    M, K, N = 640, 900, 700
    x, w = _rand(dt, (2, M, K), 7), _rand(dt, (2, K, N), 8)
    bias = _rand(dt, (N,), 9)
    want = np.stack([oracle.matmul(x[i], w[i]) for i in range(2)])
    with nc.Ctx() as ctx:
        X, W, O = ctx.from_numpy(x), ctx.from_numpy(w), ctx.zeros((2, M, N), dt)
        X0, W0, B = ctx.from_numpy(x[0]), ctx.from_numpy(w[0]), ctx.from_numpy(bias)
        C = ctx.zeros((M, N), dt)
        if resident:
            for t in (X, W, O, X0, W0, B, C):
                t.to_device()
        nc.bmm(X, W, O)
        nc.linear(X0, W0, B, C)
        if resident:
            O.to_host(), C.to_host()
        np.testing.assert_array_equal(O.numpy(), want)
        with np.errstate(over="ignore"):
            np.testing.assert_array_equal(C.numpy(), want[0] + bias)
