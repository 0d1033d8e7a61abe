"""The mid-plane field from the flutter and power tables against the oracle.

One Boris step of particles spread over the sector, inside and outside the
map's radii, for lattices on either side of each rule: fringes the flutter
table covers and a sharper one (sigmoids evaluated directly), the field index
0, a negative one, and a map coarse in r.  (With a spiral the comparison is
bound by the conditioning of s(r), a degree-6 polynomial: see the spiral
golden fixtures.)

Tolerance: the two evaluations differ by at most ~20 ulp of the field (5e-15),
which a step turns into 5e-15 times its bending (< 0.1 rad) of the velocity;
the step's own ~100 operations round to ~1e-15.  1e-14 holds both.
"""
import os
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("CUDA device required")
    from pyffa_b200 import _lib
    _lib.lib()


# fringe, field index, radial step
LATTICES = [(1.17, 7.6, 0.001), (0.2, 7.6, 0.01), (0.002, 7.6, 0.001), (1.17, 0.0, 0.001), (1.17, -0.5, 0.5)]


def lattice(fringe, k, dr):
    from pyffa_b200 import synthetic
    cfg = synthetic.lattice_bmap(r_range=(8.0, 9.3, dr), theta_step_deg=0.05)
    bm = cfg["Bmap"]
    bm["fringe_width_1"] = [0, fringe, 0, fringe, 0]
    bm["coefficients_tupel"] = [1.6 / 8.6 ** k, k]
    return cfg


@pytest.mark.parametrize("solver", ["Boris", "RK4"])
@pytest.mark.parametrize("fringe,k,dr", LATTICES)
def test_one_step_matches_oracle(fringe, k, dr, solver):
    import warnings
    from oracle import oracle as O
    from pyffa_b200 import synthetic
    from pyffa_b200.constants import FFAG_ConversionTools, FFAG_GlobalParameters
    from pyffa_b200.fields import FFAG_Bfield_analytical, FFAG_EField_new
    from pyffa_b200.track import FFAG_RungeKutta
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        bm = FFAG_Bfield_analytical(config=lattice(fringe, k, dr), max_order=0, AddNumricalMap=False)
    em = FFAG_EField_new(synthetic.emap_file(os.path.join(tempfile.mkdtemp(), "emap.txt")), EnableFlag=False)
    gp = FFAG_GlobalParameters()
    gp.AddBMap(bm)
    gp.AddEMap(em)
    n = 4000
    rng = np.random.default_rng(5)
    p = synthetic.gaussian_bunch(n, seed=3, sig_z=2e-2)
    p[:, 0] = rng.uniform(7.3, 10.2, n)           # table range 7.675 .. 9.625, direct power outside
    p[:, 4] = rng.uniform(0.0, 2 * np.pi / 12, n)
    p[:40, 4] = np.linspace(0.0, np.nextafter(2 * np.pi / 12, 0.0), 40)
    conv = FFAG_ConversionTools()
    v = conv.ConvertPrzek2Vrzek_boris(p) if solver == "Boris" else conv.ConvertPrzek2Vrzek(p)
    v[:, 7] = v[:, 8] = 1.0
    dt = synthetic.steps_per_turn_dt(steps_per_turn=720)
    ref = v.copy()
    O.track(O.Setup(bm, em, gp), solver, ref, 0.0, dt, 1)
    if solver == "Boris":
        got = v.copy()
        FFAG_RungeKutta().Boris_solve(0.0, got, dt, gp)
    else:
        got = v + FFAG_RungeKutta().rk4_step_malloc(None, 0.0, v, dt, gp)[0]
    # the velocities against their column's amplitude, the rest per element
    for c in (0, 4, 5):
        assert np.max(np.abs(got[:, c] - ref[:, c]) / np.maximum(np.abs(ref[:, c]), 1e-3)) < 1e-14, c
    for c in (1, 2, 3):
        assert np.max(np.abs(got[:, c] - ref[:, c])) < 1e-14 * np.abs(ref[:, c]).max(), c


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("fringe,m,turns", [(1.17, 1, 1 / 12), (1.17, 33, 2.05), (0.002, 33, 1 / 12)])
def test_azimuth_tracks_match_oracle(fringe, m, turns, mode):
    """Tracks without a spiral (the flutter taken a step ahead; with the
    sharp fringe evaluated directly) over a sector and past two turns, both
    stage-azimuth rules, with the trajectory and its field.  Tolerance: the
    1e-12 per sector of the spiral lattice's test."""
    import warnings
    from oracle import oracle as O
    from pyffa_b200 import seo, synthetic
    from pyffa_b200.constants import FFAG_ConversionTools, Q
    from pyffa_b200.fields import FFAG_Bfield_analytical
    cfg = synthetic.lattice_bmap(r_range=(8.0, 9.3, 0.01), theta_step_deg=0.05)
    cfg["Bmap"]["fringe_width_1"] = [0, fringe, 0, fringe, 0]
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        bm = FFAG_Bfield_analytical(config=cfg, max_order=0, AddNumricalMap=False)
    rng = np.random.default_rng(9)
    x0 = np.zeros((m, 5))
    x0[:, 0] = 8.13 + 1e-3 * rng.standard_normal(m)
    x0[:, 1] = 0.1168 + 1e-3 * rng.standard_normal(m)
    x0[:, 2:4] = 1e-3 * rng.standard_normal((m, 2))
    x0[:, 4] = FFAG_ConversionTools().Ek2P(300.0 + rng.random(m))
    t_end, cols = 2 * np.pi * turns, 7
    g1, gt, _ = seo.ThetaTracker(bm, Q).run(x0, t_end, 0.001, mode, True, cols)
    o1, ot, _ = O.ThetaTracker(bm, Q).run(x0, t_end, 0.001, mode, True, cols)
    tol = 1e-12 * max(1.0, 12 * turns)
    for c in range(4):
        assert np.abs(g1[:, c] - o1[:, c]).max() <= tol * np.abs(ot[..., c]).max(), c
    for c in range(cols):
        assert np.abs(gt[..., c] - ot[..., c]).max() <= tol * np.abs(ot[..., c]).max(), c
