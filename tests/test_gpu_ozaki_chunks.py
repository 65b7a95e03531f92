"""float64 Ozaki GEMM around the ends of its accumulation chains, for every number
of digits: one TMEM buffer with two release groups (4 digits of 128 columns, 5 to 8 of
64) or several with one, the short first chain of the second group, K just
below, at and above each.

Integers that fit the leading digits of their operand, few enough that no kept
diagonal is missing: the result is the exact sum, rounded once."""
import numpy as np
import pytest

import numc_gb300 as nc

from gpu_util import needs_gpu

pytestmark = [pytest.mark.gpu, needs_gpu]
torch = pytest.importorskip("torch")

# digits of the elements of A and B: diagonals up to p + q - 2 = S - 1
DIGITS = {1: (1, 1), 2: (2, 1), 3: (2, 2), 4: (3, 2), 5: (3, 3), 6: (4, 3), 7: (4, 4), 8: (5, 4)}


def _depths(S):
    """K of a full chain and of the second group's first one."""
    kst = 1 if S > 4 else 2 if S > 2 else 4           # 16-deep K steps of a stage
    chunk = 1024 // S // 16 // kst * kst
    return 16 * chunk, 16 * ((chunk // kst + 1) // 2 * kst)


CASES = [(S, K) for S in DIGITS for d, f in [_depths(S)]
         for K in sorted({1, f - 1, f, f + 1, d - 1, d, d + 1, d + f + 1, 2 * d, 2 * d + 1})]


def _exact(a, b):
    """a @ b of int64 matrices below 2^40 and 2^31, as Python integers."""
    parts = lambda x: ((x >> 20).astype(np.int64), (x & 0xFFFFF).astype(np.int64))  # noqa: E731
    (a1, a0), (b1, b0) = parts(a), parts(b)
    hi, mid, lo = a1 @ b1, a1 @ b0 + a0 @ b1, a0 @ b0
    return hi.astype(object) * 2 ** 40 + mid.astype(object) * 2 ** 20 + lo.astype(object)


@pytest.mark.parametrize("S,K", CASES, ids=lambda v: str(v))
def test_exact_sums(S, K):
    M, N = 130, 70
    p, q = DIGITS[S]
    rng = np.random.default_rng(100 * S + K)
    draw = lambda shape, bits: rng.integers(-(1 << bits) + 1, 1 << bits, shape)  # noqa: E731
    a, b = draw((M, K), 8 * p - 1), draw((K, N), 8 * q - 1)
    a[::7], b[:, ::5] = (1 << (8 * p - 1)) - 1, (1 << (8 * q - 1)) - 1   # sums at their largest
    out = torch.full((M, N), float("nan"), dtype=torch.float64, device="cuda")
    nc.gemm(torch.from_numpy(a.astype(np.float64)).cuda(),
            torch.from_numpy(b.astype(np.float64)).cuda(), out, algo=nc.ALGO_OZAKI, param=S)
    nc.check_status()
    want = np.array([float(v) for v in _exact(a, b).ravel()]).reshape(M, N)
    np.testing.assert_array_equal(out.cpu().numpy(), want)
