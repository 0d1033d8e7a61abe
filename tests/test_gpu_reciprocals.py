"""The push kernels' x^(-1/2) and 1 / x against 64-bit significands.

rsqrt64 refines an approximation y by y + y e (1/2 + 3/8 e), e = 1 - x y^2: the
rounding of x y^2 (2^-53) enters by a half, the last addition rounds by 2^-53, and
the series leaves 2^-58: 1.6 x 2^-53 relative.  rcp64 by y + y (e + e^2),
e = 1 - x y without rounding before the sum: 1.05 x 2^-53."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("CUDA device required")


def reciprocals(x):
    from pyffa_b200 import build
    L = ctypes.CDLL(build.build_probe())
    t = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    rs, rc = torch.empty_like(t), torch.empty_like(t)
    rc_ = L.ffa_probe_reciprocals(*(ctypes.c_void_p(a.data_ptr()) for a in (t, rs, rc)), ctypes.c_int64(t.numel()), None)
    assert rc_ == 0
    torch.cuda.synchronize()
    return rs.cpu().numpy(), rc.cpu().numpy()


@pytest.mark.parametrize("lo,hi", [(-1, 1), (-60, 60), (-1000, 1000)])
def test_within_rounding(lo, hi):
    rng = np.random.default_rng(hi)
    x = np.exp2(rng.uniform(lo, hi, 1_000_000))
    x[:4000] = np.exp2(np.round(np.linspace(lo, hi, 4000)))            # powers of two and their neighbours
    x[1000:2000] = np.nextafter(x[1000:2000], 0.0)
    x[2000:3000] = np.nextafter(x[2000:3000], np.inf)
    rs, rc = reciprocals(x)
    xl = x.astype(np.longdouble)
    assert np.abs(rs * np.sqrt(xl) - 1).max() <= 1.6 * 2.0 ** -53
    assert np.abs(rc * xl - 1).max() <= 1.05 * 2.0 ** -53
    assert np.array_equal(reciprocals(-x)[1], -rc)


def test_what_callers_keep_out():
    rs, rc = reciprocals(np.array([-1.0, -1e300, np.nan, 0.0]))
    assert np.isnan(rs).all() and np.isnan(rc[2:]).all()
