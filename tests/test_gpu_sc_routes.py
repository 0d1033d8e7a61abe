"""Routes of the space-charge update against one another and the oracle.

The plan's update reads the closed-orbit tables packed by cell when the
particles outnumber the cells, and its gather reads field pairs; the static
update takes neither.  Same values in the same order: every result is
identical, at sizes around the warp, the block, the particle pair and the
packing rule.  The open boundary's Green rows and columns on unequal grids are
held to the bounds of the square one's oracle test."""
import numpy as np
import pytest

from .test_gpu_space_charge import field_tol
from .test_zz_no_alloc import _bunch, _desc, _endpoints, _matrix, _static_update

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def seo():
    if not torch.cuda.is_available():
        pytest.skip("CUDA device required")
    from pyffa_b200 import orbit, synthetic
    t = orbit.seo_tables(synthetic.lattice_bmap(), np.linspace(290.0, 310.0, 9), nfi=361)
    return {k: t[k] for k in ("Ek_axis", "fi_axis", "r", "pr", "perimeter")}


@pytest.mark.parametrize("grid", [(5, 16, 32, 12.0), (8, 64, 64, 12.0)])
@pytest.mark.parametrize("n", [2, 31, 33, 511, 513, 2879, 2880, 2881, 40_001])   # 8 x 360 = 2880 cells
def test_plan_and_static_update_are_identical(seo, grid, n):
    from pyffa_b200.space_charge import SpaceCharge
    v = _matrix(n, n)
    a, b, keep = _bunch(v, grid, seo), _bunch(v, grid, seo), {}
    SpaceCharge(a).update(first=True)
    _static_update(b, _desc(b, seo, keep), first=True)
    assert np.array_equal(a.LocalBunch, b.LocalBunch)
    ea, eb = _endpoints(a), _endpoints(b)
    assert all(np.array_equal(ea[k], eb[k]) for k in ea)


@pytest.mark.parametrize("nx,nz", [(32, 64), (256, 16), (16, 128), (32, 32)])
def test_open_boundary_on_unequal_grids(seo, nx, nz):
    from oracle import oracle as O
    from pyffa_b200.space_charge import SpaceCharge
    v = _matrix(20_000, 3)
    marco = 1e13 / v.shape[0]
    b = _bunch(v, (6, nx, nz, 12.0), seo)
    sc = SpaceCharge(b, hockney=True)
    sc.update(first=True, roll=False)
    d, buf = sc.diag(), sc.buffers()
    m = v.copy()
    ref = O.sc_step(m, m[:, 8] != 0, seo, 6, nx, nz, 12.0, marco * 1.60217662e-19, hockney=True)
    assert np.array_equal(buf["slice_idx"], ref["slice_idx"])
    assert (buf["cell_idx"] != ref["cell_idx"]).sum() <= 2
    assert np.abs(buf["phi"] - ref["phi"]).max() <= 1e-5 * np.abs(ref["phi"]).max()
    tol = field_tol(ref["phi"], ref["ex"], ref["ez"], ref["diag"]["dx"], ref["diag"]["dz"])
    for k in ("ex", "ez"):
        assert np.abs(buf[k] - ref[k]).max() <= 4 * tol, k
