"""The z-Taylor table at every order against the oracle.  The float64 table is
laid out in planes whose widths depend on the order (4; 4 + 2; 4 + 4 + 1;
4 + 4 + 4 values a node), so every component of every order of these stacks is
another random surface, each of the same size at |z| = 5 cm, and particles sit in
the first and last cells, beside them and between.

Tolerance: a cell coordinate within an ulp of the oracle's (131 nodes: 3e-14 of
a cell) moves the interpolated field by at most ~1e-13 of its amplitude, and
a step turns that into 1e-13 times its bending (below 0.02 rad here) of the
velocity's magnitude: 2e-15, beside some 100 operations' rounding of the step.  1e-14 holds
both, as in the one-step tests of the mid-plane field."""
import os
import tempfile
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

Z = 0.05


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("CUDA device required")


def machine(order):
    from pyffa_b200 import synthetic
    from pyffa_b200.constants import FFAG_GlobalParameters
    from pyffa_b200.fields import FFAG_Bfield_analytical, FFAG_EField_new
    cfg = synthetic.lattice_bmap(r_range=(8.0, 9.3, 0.01), theta_step_deg=0.25)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        shape = FFAG_Bfield_analytical(config=cfg, max_order=0, AddNumricalMap=False)
    rng = np.random.default_rng(order)
    stacks = []
    for odd in (0, 1, 1):                                        # Bz z^2n, Bfi and Br z^(2n + 1)
        s = rng.uniform(-0.1, 0.1, (order + 1, shape.r_size, shape.fi_size))
        for n in range(order + 1):
            s[n] /= Z ** (2 * n + odd)
        stacks.append(s)
    bm = FFAG_Bfield_analytical(config=cfg, max_order=order, stacks=stacks)
    em = FFAG_EField_new(synthetic.emap_file(os.path.join(tempfile.mkdtemp(), "emap.txt")), EnableFlag=False)
    gp = FFAG_GlobalParameters()
    gp.AddBMap(bm)
    gp.AddEMap(em)
    return bm, em, gp


def rows(bm, solver):
    from pyffa_b200 import synthetic
    from pyffa_b200.constants import FFAG_ConversionTools
    n = 4000
    rng = np.random.default_rng(11)
    p = synthetic.gaussian_bunch(n, seed=3)
    dr, df = bm.r_step, bm.fi_step
    edges_r = [(bm.r_min, bm.r_min + dr), (bm.r_max - dr, bm.r_max), (bm.r_min - dr, bm.r_min), (bm.r_max, bm.r_max + dr)]
    edges_f = [(0.0, df), (bm.fi_max - df, bm.fi_max)]
    p[:, 0] = rng.uniform(bm.r_min, bm.r_max, n)
    p[:, 4] = rng.uniform(0.0, bm.fi_max, n)
    for k, (a, b) in enumerate(edges_r):
        p[100 * k:100 * k + 100, 0] = rng.uniform(a, b, 100)
    for k, (a, b) in enumerate(edges_f):
        p[50 + k:400:4, 4] = rng.uniform(a, b, 350 // 4 + 1)[:len(p[50 + k:400:4])]
    p[:, 2] = rng.choice([-1.0, 1.0], n) * rng.uniform(0.5 * Z, Z, n)
    c = FFAG_ConversionTools()
    v = c.ConvertPrzek2Vrzek_boris(p) if solver == "Boris" else c.ConvertPrzek2Vrzek(p)
    v[:, 7] = v[:, 8] = 1.0
    return v


@pytest.mark.parametrize("solver", ["Boris", "RK4"])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_one_step_matches_oracle(order, solver):
    from oracle import oracle as O
    from pyffa_b200 import synthetic
    from pyffa_b200.track import FFAG_RungeKutta
    bm, em, gp = machine(order)
    v = rows(bm, solver)
    dt = synthetic.steps_per_turn_dt(steps_per_turn=720)
    ref, flat = v.copy(), v.copy()
    O.track(O.Setup(bm, em, gp), solver, ref, 0.0, dt, 1)
    if solver == "Boris":
        got = v.copy()
        FFAG_RungeKutta().Boris_solve(0.0, got, dt, gp)
    else:
        got = v + FFAG_RungeKutta().rk4_step_malloc(None, 0.0, v, dt, gp)[0]
    # the highest order counts: without it the vertical velocities differ
    for s in (bm.Bz_stack, bm.Bfi_stack, bm.Br_stack):
        s[order] = 0.0
    O.track(O.Setup(bm, em, gp), solver, flat, 0.0, dt, 1)
    assert np.abs(flat[:, 3] - ref[:, 3]).max() > 1e-6 * np.abs(ref[:, 1]).max()
    for c in (0, 4, 5):
        assert np.max(np.abs(got[:, c] - ref[:, c]) / np.maximum(np.abs(ref[:, c]), 1e-3)) < 1e-14, c
    speed = np.hypot(np.hypot(ref[:, 1], ref[:, 3]), ref[:, 0] * ref[:, 5]).min() if solver == "Boris" else 1.9e8
    for c, scale in ((1, speed), (2, Z), (3, speed)):
        assert np.max(np.abs(got[:, c] - ref[:, c])) < 1e-14 * scale, c
