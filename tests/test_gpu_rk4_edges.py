"""FP64 RK4 at the ends of its arithmetic, against the oracle: a live particle
at rest (E equal to E0, no velocity: the azimuthal velocity is the root of an
exact 0), one without any energy, which the equations of motion make NaN, and
the field of index 0, which is B0 at every radius, at radii of either sign; and
the speed at low energies, where E0 / E is close to 1."""
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


def machine(k=7.6, B0=None, order=0):
    from pyffa_b200 import synthetic
    from pyffa_b200.constants import FFAG_GlobalParameters
    from pyffa_b200.fields import FFAG_Bfield_analytical, FFAG_EField_new
    cfg = synthetic.lattice_bmap(r_range=(8.0, 9.3, 0.01), theta_step_deg=0.05)
    cfg["Bmap"]["coefficients_tupel"] = [1.6 / 8.6 ** k if B0 is None else B0, k]
    bm = FFAG_Bfield_analytical(config=cfg, max_order=order, AddNumricalMap=False)
    em = FFAG_EField_new(synthetic.emap_file(os.path.join(tempfile.mkdtemp(), "emap.txt")), EnableFlag=False)
    gp = FFAG_GlobalParameters()
    gp.AddBMap(bm)
    gp.AddEMap(em)
    return bm, em, gp


def rows(n):
    from pyffa_b200 import synthetic
    from pyffa_b200.constants import FFAG_ConversionTools
    v = FFAG_ConversionTools().ConvertPrzek2Vrzek(synthetic.gaussian_bunch(n, seed=4))
    v[:, 7] = v[:, 8] = 1.0
    return v


def step(gp, v, dt):
    from pyffa_b200.track import FFAG_RungeKutta
    return v + FFAG_RungeKutta().rk4_step_malloc(None, 0.0, v, dt, gp)[0]


def test_particles_at_rest_and_without_energy():
    from oracle import oracle as O
    from pyffa_b200 import synthetic
    from pyffa_b200.constants import E0_J
    bm, em, gp = machine()
    v = rows(40)
    v[3, 1] = v[3, 3] = 0.0
    v[3, 5] = E0_J
    v[17, 1] = v[17, 3] = 0.0
    v[17, 5] = 0.0
    dt = synthetic.steps_per_turn_dt(steps_per_turn=720)
    ref = v.copy()
    O.track(O.Setup(bm, em, gp), "RK4", ref, 0.0, dt, 1)
    got = step(gp, v, dt)
    assert np.array_equal(ref[3, :6], v[3, :6]) and np.array_equal(got[3, :6], v[3, :6])   # it stays where it is
    assert np.isnan(ref[17, :5]).all() and np.isnan(got[17, :5]).all()
    rest = np.delete(np.arange(40), [3, 17])
    # one step of ~100 operations: see the one-step bound of the field-table test
    for c in range(6):
        assert np.max(np.abs(got[rest, c] - ref[rest, c])) <= 1e-14 * np.abs(ref[rest, c]).max(), c


def test_field_index_zero_at_any_radius():
    """The equations of motion are defined at r < 0 (fi' = v / r), and a field
    of index 0 does not depend on r."""
    from oracle import oracle as O
    from pyffa_b200 import synthetic
    bm, em, gp = machine(k=0.0, B0=1.6)
    v = rows(64)
    v[:, 0] = np.r_[-np.geomspace(1e-3, 9.0, 32), np.geomspace(1e-3, 9.0, 32)]
    v[:, 4] = np.random.default_rng(2).uniform(0, 2 * np.pi / 12, 64)
    dt = 1e-15                        # 0.3 um: the azimuth turns by at most 3e-4 rad at 1 mm
    ref = v.copy()
    O.track(O.Setup(bm, em, gp), "RK4", ref, 0.0, dt, 1)
    got = step(gp, v, dt)
    assert np.isfinite(ref[:, :6]).all() and np.isfinite(got[:, :6]).all()
    for c in range(6):
        assert np.max(np.abs(got[:, c] - ref[:, c])) <= 1e-14 * np.abs(ref[:, c]).max(), c


def test_speed_at_low_energies():
    """A straight line from its perigee: the azimuth advances by atan(v h / r).
    v^2 = c^2 (1 - (E0 / E)^2) divides the rounding of E0 / E, half an ulp of a
    number below 1 (2^-54), by beta^2: 2^-54 / beta^2 of v, half as much again
    for a square that is not fused, and ~16 ulp for the rest of the step (its
    truncation at 1e-4 rad is below 1e-16)."""
    from pyffa_b200.constants import C_LIGHT, E0_J, E0_MEV
    _, _, gp = machine(k=7.6, B0=0.0)
    n = 20_000
    v = rows(n)
    v[:, 0] = 8.5
    v[:, 1:5] = 0.0
    v[:, 5] = E0_J * (1 + np.random.default_rng(7).uniform(0.5, 10.0, n) / E0_MEV)
    ig = np.longdouble(E0_J) / v[:, 5].astype(np.longdouble)
    beta2 = 1 - ig * ig
    speed = np.longdouble(C_LIGHT) * np.sqrt(beta2)
    h = 1e-4 * 8.5 / float(speed.max())
    got = step(gp, v, h)[:, 4]
    ref = np.arctan(speed * np.longdouble(h) / np.longdouble(8.5))
    err = np.abs(got / ref - 1).astype(np.float64)
    assert (err <= 1.5 * 2.0 ** -54 / beta2.astype(np.float64) + 16 * 2.0 ** -53).all(), (err * beta2 * 2.0 ** 54).max()
