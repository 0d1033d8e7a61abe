"""Register caps of the FP64 Boris launches (chosen by warps per SM and map
order): a bunch pushed in one launch against the same bunch pushed in pieces
small enough for the small-launch cap, at the sizes around each line of the
rule.  A cap changes register allocation and at most where multiply-adds fuse:
an ulp or two (4e-16) in each of the ~20 terms that reach a column per step,
growing at most linearly over 20 steps: 20 x 20 x 4e-16 < 2e-13 of the column."""
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


@pytest.mark.parametrize("order", [0, 2, 4])
@pytest.mark.parametrize("warps,extra", [(8, 0), (8, 1), (16, 0), (16, 1), (24, 0), (24, 1), (32, 0), (32, 1), (50, 7)])
def test_one_launch_equals_pieces(order, warps, extra):
    from pyffa_b200 import synthetic
    from pyffa_b200.constants import FFAG_ConversionTools, FFAG_GlobalParameters
    from pyffa_b200.fields import FFAG_Bfield_analytical, FFAG_EField_new
    from pyffa_b200.track import Pusher, StepClock, _EphemeralBunch
    cfg = synthetic.lattice_bmap(r_range=(7.9, 9.3, 0.01), theta_step_deg=0.1)
    if order:
        bm = FFAG_Bfield_analytical(config=cfg, max_order=order, stacks=synthetic.taylor_stacks(cfg, order))
    else:
        bm = FFAG_Bfield_analytical(config=cfg, max_order=0, AddNumricalMap=False)
    em = FFAG_EField_new(synthetic.emap_file(os.path.join(tempfile.mkdtemp(), "emap.txt")), EnableFlag=True)
    gp = FFAG_GlobalParameters()
    gp.AddBMap(bm)
    gp.AddEMap(em)
    dev = torch.device("cuda", 0)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 32 * sms * warps + extra
    v = FFAG_ConversionTools().ConvertPrzek2Vrzek_boris(synthetic.gaussian_bunch(n, seed=9))
    v[:, 7] = v[:, 8] = 1.0
    dt = synthetic.steps_per_turn_dt(steps_per_turn=720)
    out = []
    for piece in (n, 32 * sms * 4):
        b = _EphemeralBunch(v, "Boris", dev)
        p = Pusher(b, gp, "Boris", "fp64", order=None)
        clock = StepClock(0.0, dt, em, "Boris", dev)
        clock.ensure(32)
        for a in range(0, n, piece):
            p.push(clock, 0, 20, 0, start=a, count=min(piece, n - a))
        torch.cuda.synchronize()
        out.append({k: b.cols[k].clone() for k in ("r", "vr", "z", "vz", "fi", "f5", "rf", "surv", "inj")})
    for k in ("surv", "inj"):
        assert torch.equal(out[0][k], out[1][k])
    for k in ("r", "vr", "z", "vz", "fi", "f5", "rf"):
        d, scale = (out[0][k] - out[1][k]).abs().max().item(), out[1][k].abs().max().item()
        assert np.isfinite(scale) and d <= 2e-13 * scale, (k, d, scale)
