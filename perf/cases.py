"""The work that users of this library have it do, as timed cases.

A case names one public entry point with its sizes, element type and options:

  host      numc_matmul on host arrays (numc's own call, copies included)
  linear    two numc_linear layers in a row on device-resident arrays
  gemm      numc_cuda_gemm on device buffers, any dtype and algorithm
  grouped   one grouped plan of many uneven float32 problems, as a CUDA graph
  rand      numc_cuda_rand_fill after numc_manual_seed

Inputs follow the distributions of the repository's own workloads: N(0, 1),
uniform [-1, 1), the row / column scaled "illscaled" and the per-element scaled
"expspread" floats, int32 in [-1000, 1000], int64 in [-2^20, 2^20], 8- and
16-bit integers over their whole range.
"""
import math

import numpy as np
import torch

import numc_gb300 as nc

DEV = "cuda"
TORCH = {"float32": torch.float32, "float64": torch.float64, "int8": torch.int8,
         "int16": torch.int16, "int32": torch.int32,
         "int64": torch.int64}
SIZE = {k: torch.empty(0, dtype=v).element_size() for k, v in TORCH.items()}
ALGOS = {"default": nc.ALGO_DEFAULT, "auto": nc.ALGO_AUTO, "simt": nc.ALGO_SIMT,
         "split16": nc.ALGO_SPLIT_FP16, "split_bf16": nc.ALGO_SPLIT_BF16,
         "ozaki": nc.ALGO_OZAKI}
# (uint8 takes int8's path, but over its whole range every output saturates.)
INT_RANGE = {"int8": (-128, 127), "int16": (-32768, 32767), "int32": (-1000, 1000),
             "int64": (-(1 << 20), 1 << 20)}
# Algorithm that numc_matmul / numc_linear use for float32 unless the program
# chooses one: numc's own FMA chains.
F32_DEFAULT = nc.ALGO_SIMT


def gemm_case(name, dtype, M, K, N, algo="default", param=-1, kind="uniform", tb=False):
    c = {"op": "gemm", "dtype": dtype, "M": M, "K": K, "N": N, "algo": algo, "param": param,
         "kind": kind, "tb": tb}
    return dict(c, name=name) if name else c


def listed():
    return [
        # numc's own call as a numc program makes it today: small host
        # matrices, default arithmetic; latency and copies count.
        {"name": "host_f32_512", "op": "host", "algo": "default", "M": 512, "K": 512, "N": 512},
        # The same call on large host matrices with the tensor-core float32
        # algorithm: copies in, product and copy out overlap.
        {"name": "host_f32_split_4096", "op": "host", "algo": "auto", "M": 4096, "K": 4096,
         "N": 4096},
        # A small MLP's forward pass, batch 256: 784 -> 128 -> 10, weights and
        # activations resident on the GPU.  The smallest device-side calls.
        {"name": "linear_f32_mlp", "op": "linear", "M": 256, "K": 784, "H": 128, "N": 10},
        # Default float32 (numc's bits) on ordinary, ragged device matrices.
        gemm_case("gemm_f32_plain", "float32", 2000, 1999, 1501, kind="normal"),
        # The precision study's size: float32 on the tensor cores.
        gemm_case("gemm_f32_split_8192", "float32", 8192, 8192, 8192, algo="split16",
                  kind="normal"),
        # Ordinary ragged float32 problem, badly scaled, B a transposed view
        # (x @ W^T).
        gemm_case("gemm_f32_split_ragged", "float32", 1536, 700, 2100, algo="auto",
                  kind="illscaled", tb=True),
        # The float64 study's size, elements spread over 2^+-20.
        gemm_case("gemm_f64_ozaki_4096", "float64", 4096, 4096, 4096, algo="ozaki", param=8,
                  kind="expspread"),
        # Integer workloads: exact, modulo 2^bits.
        gemm_case("gemm_i32_1024", "int32", 1024, 1024, 1024),
        gemm_case("gemm_i64_ragged", "int64", 1500, 1024, 1111),
        gemm_case("gemm_i8_4096", "int8", 4096, 4096, 4096),
        # Batched uneven problems in one plan, and MLP chains' first layers.
        {"name": "grouped_f32_2048", "op": "grouped", "problems": 2048, "chains": 256,
         "lo": 16, "hi": 1024},
        # Random inputs generated on the GPU, 256 MiB.
        {"name": "rand_f32_64Mi", "op": "rand", "dtype": "float32", "n": 64 << 20},
    ]


def _log(rng, lo, hi):
    """An integer in [lo, hi], spread over its logarithm; every third one is
    a multiple of 64 where there is one."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 1 / 3 and v >= 64:
        v = v // 64 * 64
    return max(lo, min(hi, v))


def draw(rng):
    op = rng.choice(["host", "host_split", "linear", "f32", "split", "f64", "int", "int", "int8",
                     "grouped", "rand"])
    tb = rng.random() < 0.3
    if op == "host":
        return {"op": "host", "algo": "default", "M": _log(rng, 64, 1024),
                "K": _log(rng, 64, 1024), "N": _log(rng, 64, 1024)}
    if op == "host_split":
        return {"op": "host", "algo": "auto", "M": _log(rng, 1024, 4096),
                "K": _log(rng, 512, 4096), "N": _log(rng, 1024, 4096)}
    if op == "linear":
        return {"op": "linear", "M": _log(rng, 16, 1024), "K": _log(rng, 64, 1024),
                "H": _log(rng, 32, 512), "N": _log(rng, 8, 128)}
    if op == "f32":
        return gemm_case(None, "float32", _log(rng, 128, 2560), _log(rng, 128, 2560),
                         _log(rng, 128, 2560), kind=rng.choice(["normal", "uniform"]), tb=tb)
    if op == "split":
        return gemm_case(None, "float32", _log(rng, 256, 8192), _log(rng, 128, 8192),
                         _log(rng, 256, 8192), algo="auto",
                         kind=rng.choice(["normal", "illscaled"]), tb=tb)
    if op == "f64":
        return gemm_case(None, "float64", _log(rng, 256, 4096), _log(rng, 256, 4096),
                         _log(rng, 256, 4096), algo="ozaki", param=rng.randint(4, 8),
                         kind=rng.choice(["uniform", "expspread"]), tb=tb)
    if op == "int":
        return gemm_case(None, rng.choice(["int16", "int32", "int64"]), _log(rng, 128, 2048),
                         _log(rng, 128, 2048), _log(rng, 128, 2048), tb=tb)
    if op == "int8":
        return gemm_case(None, "int8", _log(rng, 256, 4096), _log(rng, 256, 4096),
                         _log(rng, 256, 4096), tb=tb)
    if op == "grouped":
        return {"op": "grouped", "problems": _log(rng, 64, 2048), "chains": rng.randint(0, 256),
                "lo": 16, "hi": _log(rng, 256, 1024)}
    return {"op": "rand", "dtype": rng.choice(["float32", "float64", "int8", "int32"]),
            "n": _log(rng, 1000, 32 << 20)}


# ---- inputs ------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _uniform(gen, shape, dtype):
    return torch.rand(shape, device=DEV, generator=gen, dtype=dtype) * 2 - 1


def _matrix(gen, shape, dtype, kind):
    t = TORCH[dtype]
    if dtype in INT_RANGE:
        lo, hi = INT_RANGE[dtype]
        return torch.randint(lo, hi + 1, shape, device=DEV, generator=gen, dtype=t)
    if kind == "normal":
        return torch.randn(shape, device=DEV, generator=gen, dtype=t)
    x = _uniform(gen, shape, t)
    if kind == "expspread":
        e = torch.randint(-20, 21, shape, device=DEV, generator=gen, dtype=torch.int32)
        x = torch.ldexp(x, e)
    return x


def _operands(c, seed):
    """(A, B) of a gemm case; B a transposed view when c["tb"]."""
    gen = _gen(seed)
    M, K, N = c["M"], c["K"], c["N"]
    kind = "normal" if c["kind"] == "illscaled" else c["kind"]
    a = _matrix(gen, (M, K), c["dtype"], kind)
    b = _matrix(gen, (N, K) if c["tb"] else (K, N), c["dtype"], kind)
    if c["tb"]:
        b = b.t()
    if c["kind"] == "illscaled":
        u = 10.0 ** (torch.rand(M, device=DEV, generator=gen, dtype=torch.float64) * 8 - 4)
        v = 10.0 ** (torch.rand(N, device=DEV, generator=gen, dtype=torch.float64) * 8 - 4)
        a = (a * u[:, None]).to(a.dtype)
        b = (b * v[None, :]).to(a.dtype)
        if c["tb"]:
            b = b.t().contiguous().t()
    return a, b


def _host_operands(c, seed):
    gen = _gen(seed)
    return (_uniform(gen, (c["M"], c["K"]), torch.float32),
            _uniform(gen, (c["K"], c["N"]), torch.float32))


def _linear_operands(c, seed):
    gen = _gen(seed)
    x = _uniform(gen, (c["M"], c["K"]), torch.float32)
    w1 = torch.randn((c["K"], c["H"]), device=DEV, generator=gen) * 0.05
    b1 = torch.randn((c["H"],), device=DEV, generator=gen) * 0.05
    w2 = torch.randn((c["H"], c["N"]), device=DEV, generator=gen) * 0.05
    b2 = torch.randn((c["N"],), device=DEV, generator=gen) * 0.05
    return x, w1, b1, w2, b2


def _grouped_dims(c, seed):
    """(M, K, N) of every problem: log-uniform sizes, then the MLP layers."""
    rng = np.random.default_rng(seed)
    d = np.exp(rng.uniform(np.log(c["lo"]), np.log(c["hi"]), (c["problems"], 3)))
    dims = [tuple(int(v) for v in row) for row in d.round().astype(int)]
    return dims + [(256, 784, 128)] * c["chains"]


def _grouped_operands(c, seed):
    """Every problem's (a, b, out) as views of three flat buffers (256-byte
    aligned each) and the flat output buffer."""
    # the sizes of a workload are fixed; its values change with the seed
    dims = _grouped_dims(c, 42)
    up = lambda n: (n + 63) // 64 * 64  # noqa: E731
    gen = _gen(seed)
    fa = _uniform(gen, (sum(up(m * k) for m, k, n in dims),), torch.float32)
    fb = _uniform(gen, (sum(up(k * n) for m, k, n in dims),), torch.float32)
    fo = torch.zeros(sum(up(m * n) for m, k, n in dims), device=DEV)
    pa = pb = po = 0
    probs = []
    for m, k, n in dims:
        probs.append((fa[pa:pa + m * k].view(m, k), fb[pb:pb + k * n].view(k, n),
                      fo[po:po + m * n].view(m, n)))
        pa, pb, po = pa + up(m * k), pb + up(k * n), po + up(m * n)
    return probs, fo


# ---- states ------------------------------------------------------------------


class State:
    """What a program keeps between calls: arrays, buffers, a context or plan."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


class Owner:
    """A context that is freed with the last array or view that refers to it."""

    def __init__(self):
        self.ctx = nc.Ctx()

    def __del__(self):
        self.ctx.free()


class _HostView:
    """numpy's view of a contiguous float32 Array's host buffer, no copy."""

    def __init__(self, arr, owner):
        self.owner = owner
        self.__array_interface__ = {"data": (nc.lib().numc_array_data(arr.ptr), False),
                                    "shape": arr.shape, "typestr": "<f4", "version": 3}


class _DeviceView:
    """torch's view of a resident contiguous float32 Array, no copy."""

    def __init__(self, arr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (arr.device_ptr(), False), "shape": arr.shape,
                                         "typestr": "<f4", "version": 3}


def _resident(ctx, t):
    return ctx.from_numpy(t.cpu().numpy()).to_device()


def prepare(case, seed):
    op = case["op"]
    if op == "host":
        nc.set_algo("float32", ALGOS[case["algo"]] if case["algo"] != "default" else F32_DEFAULT)
        owner = Owner()
        ctx = owner.ctx
        a, b = _host_operands(case, seed)
        A, B = ctx.from_numpy(a.cpu().numpy()), ctx.from_numpy(b.cpu().numpy())
        C = ctx.zeros((case["M"], case["N"]), "float32")
        return State(op=op, owner=owner, a=A, b=B, out=C, view=np.asarray(_HostView(C, owner)))
    if op == "linear":
        nc.set_algo("float32", F32_DEFAULT)
        owner = Owner()
        ctx = owner.ctx
        x, w1, b1, w2, b2 = (_resident(ctx, t) for t in _linear_operands(case, seed))
        h = ctx.zeros((case["M"], case["H"]), "float32").to_device()
        y = ctx.zeros((case["M"], case["N"]), "float32").to_device()
        views = [torch.as_tensor(_DeviceView(v, owner), device=DEV) for v in (h, y)]
        return State(op=op, owner=owner, x=x, w1=w1, b1=b1, w2=w2, b2=b2, h=h, y=y, views=views)
    if op == "gemm":
        a, b = _operands(case, seed)
        algo, param = ALGOS[case["algo"]], case["param"]
        need = nc.workspace_size(case["dtype"], algo, param, case["M"], case["K"], case["N"])
        ws = torch.empty(need, dtype=torch.uint8, device=DEV) if need else None
        out = torch.zeros((case["M"], case["N"]), dtype=a.dtype, device=DEV)
        return State(op=op, a=a, b=b, out=out, algo=algo, param=param, ws=ws)
    if op == "grouped":
        probs, flat = _grouped_operands(case, seed)
        return State(op=op, plan=nc.GemmPlan(probs, nc.ALGO_SPLIT_FP16), flat=flat)
    return State(op=op, seed=seed,
                 out=torch.empty(case["n"], dtype=TORCH[case["dtype"]], device=DEV))


def run(state):
    op = state.op
    if op == "host":
        nc.matmul(state.a, state.b, state.out)
        return state.view
    if op == "linear":
        nc.linear(state.x, state.w1, state.b1, state.h)
        nc.linear(state.h, state.w2, state.b2, state.y)
        return state.views
    if op == "gemm":
        nc.gemm(state.a, state.b, state.out, algo=state.algo, param=state.param,
                workspace=state.ws)
        return state.out
    if op == "grouped":
        state.plan.run(graph=True)
        return state.flat
    nc.manual_seed(state.seed)
    nc.rand_fill(state.out)
    return state.out


# ---- what a pass cannot do without, and its exact results ----------------------


def work(case):
    op = case["op"]
    if op == "rand":
        return {"bytes": case["n"] * SIZE[case["dtype"]], "flops": 0}
    if op == "grouped":
        dims = _grouped_dims(case, 42)
        return {"bytes": 4 * sum(m * k + k * n + m * n for m, k, n in dims),
                "flops": 2 * sum(m * k * n for m, k, n in dims)}
    M, K, N = case["M"], case["K"], case["N"]
    if op == "linear":
        H = case["H"]
        return {"bytes": 4 * (M * K + K * H + 2 * H + M * H + H * N + N + M * N),
                "flops": 2 * M * H * (K + N)}
    size = SIZE[case.get("dtype", "float32")]
    return {"bytes": size * (M * K + K * N + M * N), "flops": 2 * M * K * N}


def exact(case, seed):
    op = case["op"]
    if op == "host":
        a, b = _host_operands(case, seed)
        return (a.double() @ b.double()).cpu().numpy()
    if op == "linear":
        x, w1, b1, w2, b2 = (t.double() for t in _linear_operands(case, seed))
        h = x @ w1 + b1
        return [h, h @ w2 + b2]
    if op == "grouped":
        probs, flat = _grouped_operands(case, seed)
        out = torch.zeros_like(flat, dtype=torch.float64)
        base = flat.data_ptr()
        for a, b, o in probs:
            p = (o.data_ptr() - base) // 4
            out[p:p + o.numel()] = (a.double() @ b.double()).reshape(-1)
        return out
    if op == "gemm" and case["dtype"] in ("float32", "float64"):
        a, b = _operands(case, seed)
        return a.double() @ b.double()
    if op == "gemm" and case["dtype"] in ("int16", "int32", "int64"):
        # |sums| stay below 2^53 over the declared ranges
        a, b = _operands(case, seed)
        return (a.double() @ b.double()).to(torch.int64).to(a.dtype)
    return None   # 8-bit stores follow numc's build; random bytes have no such value
