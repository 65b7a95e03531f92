"""The scale + split pass that stages rows in shared memory: every change of rows
per block and of copy (bulk, pairs, single elements, across columns) over the
edges of K, through single GEMMs and grouped plans, against the general two-pass
split: the same product with K padded by zeros beyond the staged range has the
same planes and the same sums, bit for bit."""
import numpy as np
import pytest

import numc_gb300 as nc
from numc_gb300 import synth

from gpu_util import needs_gpu

pytestmark = [pytest.mark.gpu, needs_gpu]
torch = pytest.importorskip("torch")

KS = [1, 2, 3, 63, 64, 65, 255, 256, 257, 512, 513, 1023, 1024, 1025, 1536, 1537]


def layouts(x):
    """The same matrix dense, off by one element, with padded rows (odd and even),
    transposed, and with a column step."""
    R, K = x.shape
    t = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    yield t
    flat = torch.zeros(R * K + 1, device="cuda")
    flat[1:] = t.reshape(-1)
    yield flat[1:].reshape(R, K)
    for pad in (1, 2):
        wide = torch.full((R, K + pad), float("nan"), device="cuda")
        wide[:, :K] = t
        yield wide[:, :K]
    yield t.t().contiguous().t()
    step = torch.full((R, 2 * K), float("nan"), device="cuda")
    step[:, ::2] = t
    yield step[:, ::2]


def run(ta, tb, grouped):
    out = torch.full((ta.shape[0], tb.shape[1]), float("nan"), device="cuda")
    if grouped:
        plan = nc.GemmPlan([(ta, tb, out)], nc.ALGO_SPLIT_FP16, 128)
        plan.run()
    else:
        nc.gemm(ta, tb, out, algo=nc.ALGO_SPLIT_FP16)
    nc.check_status()
    return out.cpu().numpy()


@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("K", KS)
def test_layouts_give_the_same_bits(K, grouped):
    M, N = 133, 70
    a, b = synth.operands("uniform", M, K, N, dtype="float32", seed=K)
    a[5] = 0.0                       # a row of zeros, a subnormal row, a huge row
    a[6] *= np.float32(1e-38)
    a[7] *= np.float32(1e30)
    pad = 1600 - K
    want = run(torch.from_numpy(np.pad(a, ((0, 0), (0, pad)))).cuda(),
               torch.from_numpy(np.pad(b, ((0, pad), (0, 0)))).cuda(), grouped)
    assert np.isfinite(want).all() and not want[5].any()
    for ta, tb in zip(layouts(a), layouts(b)):
        np.testing.assert_array_equal(run(ta, tb, grouped), want)


@pytest.mark.parametrize("K", [40, 300, 700, 1300])
def test_nonfinite_rows_are_recomputed(K):
    a, b = synth.operands("uniform", 300, K, 90, dtype="float32", seed=K)
    a[299, K - 1] = np.inf
    b[0, 89] = np.nan
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    single, plain = torch.empty(300, 90, device="cuda"), torch.empty(300, 90, device="cuda")
    nc.gemm(ta, tb, single, algo=nc.ALGO_SPLIT_FP16)
    plan = nc.GemmPlan([(ta, tb, plain)], nc.ALGO_SPLIT_FP16, 64)
    plan.run()
    nc.check_status()
    for got in (single.cpu().numpy(), plain.cpu().numpy()):
        assert np.isnan(got[:, 89]).all()
        assert np.isinf(got[299, :89]).all() and np.isfinite(got[:299, :89]).all()
