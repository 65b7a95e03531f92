"""CTA-pair tiles narrower than 256 columns (160 to 224, picked where they round
better over the device): the split products store the bits of 256-column
tiles, int8 the bytes of the CUDA-core kernel, with ragged last tiles and a
non-finite column beside a tile's edge."""
import hashlib
import os
import subprocess
import sys

import numpy as np
import pytest

import numc_gb300 as nc
from gpu_util import needs_gpu

pytestmark = [pytest.mark.gpu, needs_gpu]
torch = pytest.importorskip("torch")

# (M, N) with 224-, 192- and 160-column tiles on 76 pairs, ragged and not
SIZES = [(4096, 1120), (4000, 4096), (3000, 2500), (2500, 2600), (4096, 4100), (2049, 3071)]

_SCRIPT = r"""
import sys, hashlib, torch, numc_gb300 as nc
g = torch.Generator(device="cuda").manual_seed(3)
for M, N in %r:
    a = torch.randn(M, 200, device="cuda", generator=g)
    b = torch.randn(200, N, device="cuda", generator=g)
    for algo, param in ((nc.ALGO_SPLIT_FP16, 0), (nc.ALGO_SPLIT_BF16, 3)):
        c = torch.full((M, N), float("nan"), device="cuda")
        nc.gemm(a, b, c, algo=algo, param=param)
        nc.check_status()
        print(M, N, algo, hashlib.md5(c.cpu().numpy().tobytes()).hexdigest())
""" % (SIZES,)


def test_split_bits_do_not_depend_on_the_width():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    outs = []
    for tile in (None, "256"):
        env = dict(os.environ)
        if tile:
            env["NUMC_CUDA_SPLIT_TILE"] = tile
        r = subprocess.run([sys.executable, "-c", _SCRIPT], env=env, cwd=root,
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr
        outs.append(r.stdout)
    assert outs[0] == outs[1] and outs[0].count("\n") == 2 * len(SIZES)


@pytest.mark.parametrize("profile", [nc.INT8_X86_AVX2, nc.INT8_ARM_NEON])
@pytest.mark.parametrize("dt", ["int8", "uint8"])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_int8_bytes(size, dt, profile):
    M, N = size
    t = getattr(torch, dt)
    g = torch.Generator(device="cuda").manual_seed(4)
    lo, hi = (-12, 13) if dt == "int8" else (0, 3)
    a = torch.randint(lo, hi, (M, 600), device="cuda", generator=g, dtype=t)
    b = torch.randint(lo, hi, (600, N), device="cuda", generator=g, dtype=t)
    c, d = torch.zeros((2, M, N), device="cuda", dtype=t)
    nc.gemm(a, b, c, algo=nc.ALGO_TC_INT8, param=profile)
    nc.gemm(a, b, d, algo=nc.ALGO_SIMT, param=profile)
    nc.check_status()
    assert torch.equal(c, d)


def test_non_finite_column_at_a_tile_edge():
    M, K, N = 4096, 150, 4096            # 224-column tiles
    g = torch.Generator(device="cuda").manual_seed(5)
    a = torch.randn(M, K, device="cuda", generator=g)
    b = torch.randn(K, N, device="cuda", generator=g)
    b[3, 224] = float("inf")
    b[5, 447] = float("nan")
    c = torch.zeros((M, N), device="cuda")
    nc.gemm(a, b, c, algo=nc.ALGO_SPLIT_FP16)
    nc.check_status()
    want = a.double() @ b.double()
    bad = ~torch.isfinite(want)
    assert torch.equal(torch.isfinite(c), torch.isfinite(want))
    assert bad.any(dim=0).nonzero().flatten().tolist() == [224, 447]
    scale = a.abs().double() @ b.nan_to_num(0, 0, 0).abs().double()
    err = ((c.double() - want).abs() / scale)[~bad].max().item()
    assert err <= 4 * 2.0 ** -22 + 2 * (3 * K + 2) * 2.0 ** -24
