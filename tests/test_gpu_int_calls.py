"""16- to 64-bit integer products of a context's arrays, which take the tensor
cores where those are faster: resident calls only enqueue work, a batch takes
them as one product does, and failures and refused memory stay with the context
that met them."""
import numpy as np
import pytest

import numc_gb300 as nc
import oracle

from gpu_util import needs_gpu

pytestmark = [pytest.mark.gpu, needs_gpu]
torch = pytest.importorskip("torch")

DTYPES = ["int16", "int32", "int64"]
LIMIT_NS = 20_000_000   # 20 ms per abandoned wait


def _rand(dt, shape, seed):
    info = np.iinfo(dt)
    return np.random.default_rng(seed).integers(info.min, info.max, shape, dtype=dt, endpoint=True)


class starved_waits:
    """Bounded waits run out after LIMIT_NS: the producers issue no loads."""

    def __enter__(self):
        torch.cuda.synchronize()
        nc.lib().numc_cuda_debug_wait_timeout(LIMIT_NS, 1)

    def __exit__(self, *exc):
        torch.cuda.synchronize()
        nc.lib().numc_cuda_debug_wait_timeout(0, 0)


def _internal(call):
    with pytest.raises(nc.NumcError) as ei:
        call()
    assert ei.value.code == nc.ERR_INTERNAL
    assert "bounded wait" in ei.value.msg


def _call(op, ctx, dt, n, resident):
    """(call, output array, expected result) of an n^3 product or two of them."""
    if op == "bmm":
        x, w = _rand(dt, (2, n, n), 1), _rand(dt, (2, n, n), 2)
        want = np.stack([oracle.matmul(x[i], w[i]) for i in range(2)])
    else:
        x, w = _rand(dt, (n, n), 1), _rand(dt, (n, n), 2)
        want = oracle.matmul(x, w)
    X, W, O = ctx.from_numpy(x), ctx.from_numpy(w), ctx.zeros(want.shape, dt)
    bias = ctx.from_numpy(np.ones(n, dt)) if op == "linear" else None
    if bias is not None:
        with np.errstate(over="ignore"):
            want = want + np.ones(n, dt)
    if resident:
        for t in (X, W, O) + ((bias,) if bias else ()):
            t.to_device()
    fn = {"matmul": nc.matmul, "dot": nc.dot, "bmm": nc.bmm}.get(op)
    return (lambda: fn(X, W, O) if fn else nc.linear(X, W, bias, O)), O, want


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("op", ["matmul", "linear", "bmm", "dot"])
def test_resident_calls_only_enqueue(op, dt):
    with nc.Ctx() as ctx:
        call, out, want = _call(op, ctx, dt, 1024, True)
        call()                  # scratch grows to its size here
        ctx.synchronize()
        s = torch.cuda.ExternalStream(ctx.stream())
        with torch.cuda.stream(s):
            torch.cuda._sleep(400_000_000)   # about 0.2 s
        n = nc.launch_count()
        call()
        assert not s.query(), "the call waited for its stream"
        assert nc.launch_count() - n == (4 if op == "bmm" else 2)   # the tensor cores' two
        out.to_host()
        np.testing.assert_array_equal(out.numpy(), want)


@pytest.mark.parametrize("resident", [False, True])
def test_failures_of_other_streams_stay_there(resident):
    """An integer product neither reports nor clears what another stream's kernel
    recorded."""
    a = torch.rand((300, 520), device="cuda")
    b = torch.rand((520, 270), device="cuda")
    c = torch.zeros((300, 270), device="cuda")
    with nc.Ctx() as ctx:
        call, out, want = _call("matmul", ctx, "int32", 1024, resident)
        with starved_waits():
            nc.gemm(a, b, c, algo=nc.ALGO_SPLIT_FP16)
        call()
        out.to_host()
        np.testing.assert_array_equal(out.numpy(), want)
        _internal(nc.check_status)
        nc.check_status()


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("op", ["matmul", "linear", "bmm", "dot"])
def test_host_call_reports_its_own_failure(op, dt):
    with nc.Ctx() as ctx, nc.Ctx() as other:
        call, out, want = _call(op, ctx, dt, 640, False)
        call2, out2, want2 = _call("matmul", other, dt, 640, False)
        with starved_waits():
            _internal(call)
        call2()
        np.testing.assert_array_equal(out2.numpy(), want2)
        call()
        np.testing.assert_array_equal(out.numpy(), want)
        nc.check_status()


@pytest.mark.parametrize("where", ["to_host", "synchronize", "check_status", "host_call"])
def test_resident_call_reports_at_the_next_wait(where):
    with nc.Ctx() as ctx:
        call, out, want = _call("matmul", ctx, "int32", 1024, True)
        small = ctx.from_numpy(np.eye(1024, 4, dtype="int32"))   # a CUDA-core product
        res = ctx.zeros((1024, 4), "int32")
        with starved_waits():
            call()
        wait = {"to_host": out.to_host, "synchronize": ctx.synchronize,
                "check_status": nc.check_status, "host_call": lambda: nc.matmul(out, small, res)}
        _internal(wait[where])
        call()
        wait[where]()
        out.to_host()
        np.testing.assert_array_equal(out.numpy(), want)
        nc.check_status()


def test_resident_batch_takes_the_tensor_cores():
    """8 products that gain a few us each."""
    n, P = 512, 8
    x, w = _rand("int32", (P, n, n), 3), _rand("int32", (P, n, n), 4)
    with nc.Ctx() as ctx:
        X, W, O = ctx.from_numpy(x), ctx.from_numpy(w), ctx.zeros((P, n, n), "int32")
        for t in (X, W, O):
            t.to_device()
        k = nc.launch_count()
        nc.bmm(X, W, O)
        assert nc.launch_count() - k == 2 * P
        O.to_host()
        np.testing.assert_array_equal(O.numpy(), np.stack([oracle.matmul(x[i], w[i]) for i in range(P)]))


def test_no_room_for_the_digits():
    """The device refuses the digits' memory: the context keeps the scratch that it
    has, the CUDA cores take the call, and the next one does not ask again."""
    n = 640
    a, b = _rand("int32", (n, n), 5), _rand("int32", (n, n), 6)
    want = oracle.matmul(a, b)
    with nc.Ctx() as ctx:
        A, B, C = ctx.from_numpy(a), ctx.from_numpy(b), ctx.zeros((n, n), "int32")
        nc.matmul_naive(A, B, C)          # scratch for the staged operands alone
        nc.lib().numc_cuda_debug_fail_malloc(1000)
        try:
            for _ in range(2):
                C.write(np.zeros_like(want))
                k = nc.launch_count()
                nc.matmul(A, B, C)
                assert nc.launch_count() - k == 1
                np.testing.assert_array_equal(C.numpy(), want)
            # one allocation would fail, and the call makes none
            nc.lib().numc_cuda_debug_fail_malloc(1)
            nc.matmul(A, B, C)
            with pytest.raises(nc.NumcError) as ei:
                A.to_device()
            assert ei.value.code == nc.ERR_MALLOC
        finally:
            nc.lib().numc_cuda_debug_fail_malloc(0)


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("shape", [(640, 640, 640), (1, 9001, 1), (64, 5000, 64)],
                         ids=lambda s: "x".join(map(str, s)))
def test_gemm_reports_abandoned_waits(dt, shape):
    """numc_cuda_gemm with a workspace: one K split and several (which add into a
    cleared output)."""
    M, K, N = shape
    a, b = _rand(dt, (M, K), 7), _rand(dt, (K, N), 8)
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    need = nc.workspace_size(dt, nc.ALGO_DEFAULT, -1, M, K, N)
    if not need:
        pytest.skip("the CUDA cores take this problem")
    ws = torch.zeros(need, dtype=torch.uint8, device="cuda")
    out = torch.zeros((M, N), dtype=ta.dtype, device="cuda")
    with starved_waits():
        nc.gemm(ta, tb, out, workspace=ws)
        _internal(nc.check_status)
    nc.check_status()
    nc.gemm(ta, tb, out, workspace=ws)
    nc.check_status()
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.matmul(a, b))


def test_captured_call_takes_the_cuda_cores():
    """A graph outlives the scratch of the calls captured in it: no digits there."""
    n = 1024
    a, b = _rand("int32", (n, n), 9), _rand("int32", (n, n), 10)
    with nc.Ctx() as ctx:
        A, B, Z = ctx.from_numpy(a), ctx.from_numpy(b), ctx.zeros((n, n), "int32")
        C = ctx.zeros((n, n), "int32")
        for t in (A, B, Z, C):
            t.to_device()
        nc.matmul(A, B, C)
        ctx.synchronize()
        g = torch.cuda.CUDAGraph()
        k = nc.launch_count()
        with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(ctx.stream())):
            nc.matmul(A, B, C)
        assert nc.launch_count() - k == 1
        nc.matmul(Z, B, C)              # zeros in the output
        ctx.synchronize()
        g.replay()
        torch.cuda.synchronize()
        C.to_host()
        np.testing.assert_array_equal(C.numpy(), oracle.matmul(a, b))
