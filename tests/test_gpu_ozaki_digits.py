"""float64 Ozaki products at the limits of their digit sums: the bound of s
digits, (s + 3) K 2^-8s 2^(e_i + f_j) plus the rounding of the result."""
import numpy as np
import pytest

import numc_gb300 as nc

from gpu_util import needs_gpu

pytestmark = [pytest.mark.gpu, needs_gpu]
torch = pytest.importorskip("torch")


def test_ozaki_extreme_digits_and_long_k():
    """float64: digits that are all -128 (sums beyond the fast conversion),
    and K past 2^24, where A's digits leave headroom (sums of ones: exact)."""
    a = np.full((130, 1030), -1082163328.0)   # -0x40808080: digits -64, -128, ...
    b = np.full((1030, 70), -1082163328.0)
    out = torch.zeros((130, 70), dtype=torch.float64, device="cuda")
    for s in (4, 5, 8):
        nc.gemm(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), out, algo=nc.ALGO_OZAKI,
                param=s)
        nc.check_status()
        exact = 1030 * 1082163328 ** 2
        # (s + 3) K 2^-8s 2^(31 + 31) for the digits, 2^-53 for the rounding
        bound = (s + 3) * 1030 * 2.0 ** (62 - 8 * s) + 2.0 ** -53 * exact
        assert np.abs(out.cpu().numpy() - float(exact)).max() <= bound
    k = (1 << 24) + 5
    x = torch.ones((1, k), dtype=torch.float64, device="cuda")
    y = torch.ones((k, 1), dtype=torch.float64, device="cuda")
    out = torch.zeros((1, 1), dtype=torch.float64, device="cuda")
    nc.gemm(x, y, out, algo=nc.ALGO_OZAKI, param=8)
    nc.check_status()
    assert out.item() == k
