"""numc_array_rand's fill at the edges of its runs, rows and blocks, byte for
byte against the oracle: lengths around a run, a warp's 4 KiB rows, a block,
the 1 MiB layout threshold, and every run length of the large fill."""
import threading

import pytest

import numc_gb300 as nc
import oracle
from gpu_util import needs_gpu

pytestmark = [pytest.mark.gpu, needs_gpu]
torch = pytest.importorskip("torch")

MIB = 1 << 20
SMALL = [1, 3, 4, 127, 128, 129, 511, 4 * 32 * 64 - 1, 4 * 32 * 64, 4 * 32 * 64 + 5, 70001]
CASES = ([(dt, n) for dt in ("int8", "int16", "float32", "float64") for n in SMALL] +
         [("int8", 4 * 128 * 64 * 3 + 2), ("int8", MIB), ("int8", MIB + 1), ("float32", MIB // 4),
          ("float32", MIB // 4 + 1), ("float32", 300001), ("int16", 5 * MIB + 3),
          ("float32", 5 * MIB + 3), ("float64", 10 * MIB + 1), ("int32", 20 * MIB + 7),
          ("int8", 41 * MIB + 9)])


@pytest.mark.parametrize("dt,n", CASES, ids=[f"{d}-{n}" for d, n in CASES])
def test_edges_match_oracle(dt, n):
    def body(box):
        nc.manual_seed(n)
        for off in (0, 1):    # the second fill continues the state, unaligned
            t = torch.full((n + off,), 7, device="cuda").to(getattr(torch, dt))
            nc.rand_fill(t[off:])
            torch.cuda.synchronize()
            box.append(t[off:].cpu().numpy())
    nc.rand_set_threads(6)
    box = []
    try:
        th = threading.Thread(target=body, args=(box,))   # the state is per thread
        th.start()
        th.join()
    finally:
        nc.rand_set_threads(0)
    st = oracle.rand_seed(n)
    assert len(box) == 2
    for got in box:
        assert got.tobytes() == oracle.rand(dt, (n,), st, 6).tobytes()
