"""The per-loop reductions where a thread takes a run of values and blocks
combine through integer atomics (GPU)."""
import math
import sys

import numpy as np
import pytest

from mgcfd import ops

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

N = 400_001  # more than 608 blocks of 256 threads hold at one value each
BLOCK = 256


def _values(kind):
    rng = np.random.default_rng(3)
    x = np.exp(rng.uniform(-60, 60, N))
    if kind == "negative in one block":
        x[5 * BLOCK + 17] = -1e-300
    elif kind == "both signs":
        x *= rng.choice([-1.0, 1.0], N)
    elif kind == "negative":
        x = -x
    elif kind == "negative last":
        x[-1] = -3.0
    elif kind == "negative zero":
        x[rng.integers(0, N, 20)] = -0.0
    elif kind == "zeros and a negative subnormal":
        x[:] = 0.0
        x[N // 2] = -5e-324
    elif kind == "infinite":
        x[rng.random(N) < 0.5] = np.inf
    elif kind == "minus infinity":
        x[N // 3] = -np.inf
    elif kind == "nan among others":
        x[rng.random(N) < 0.9] = np.nan
    elif kind == "all nan":
        x[:] = np.nan
    elif kind == "all infinite":
        x[:] = np.inf
    elif kind == "largest":
        x[:] = sys.float_info.max
    elif kind == "just below the largest":
        x[:] = sys.float_info.max
        x[77] = np.nextafter(sys.float_info.max, 0)
    return x


@pytest.mark.parametrize("n", [1, BLOCK + 1, N])
@pytest.mark.parametrize("kind", ["positive", "negative in one block", "both signs", "negative", "negative last",
                                  "negative zero", "zeros and a negative subnormal", "infinite", "minus infinity",
                                  "nan among others", "all nan", "all infinite", "largest", "just below the largest"])
def test_get_min_dt(kind, n):
    """get_min_dt_kernel (time_stepping_kernels.h:34-41) keeps its DBL_MAX start
    unless dt < it: exact, NaN never taken."""
    x = _values(kind)[-n:].copy()
    want = min([sys.float_info.max] + [v for v in x.tolist() if v < sys.float_info.max])
    out = torch.full((1,), 7.0, dtype=torch.float64, device="cuda")
    dt = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    ops.get_min_dt(n, dt.data_ptr(), out.data_ptr())
    torch.cuda.synchronize()
    assert out.item() == want


@pytest.mark.parametrize("n", [1, 51, N])
def test_calc_rms_and_count_bad_vals(n):
    """calc_rms adds the sum of squares: positive terms, in runs of 13, a tree of 13
    steps and up to 608 atomics, so within 640 2^-53 of itself; count_bad_vals
    (validation.h:102-115) is exact and adds to what is there."""
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 5)) * np.exp(rng.uniform(-20, 5, (n, 5)))
    res = torch.from_numpy(x).cuda()
    rms = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ops.calc_rms(n, res.data_ptr(), rms.data_ptr())
    torch.cuda.synchronize()
    want = math.fsum((x * x).ravel().tolist())
    assert abs(rms.item() - want) <= 640 * 2.0 ** -53 * want
    bad = x.copy().reshape(-1)
    at = rng.choice(5 * n, min(5 * n, 2999), replace=False)
    bad[at] = rng.choice([np.nan, np.inf, -np.inf], len(at))
    var = torch.from_numpy(bad).cuda()
    count = torch.full((1,), 3, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ops.count_bad_vals(n, var.data_ptr(), count.data_ptr())
    torch.cuda.synchronize()
    assert count.item() == 3 + len(at)
