"""The builds of the float64 pushers that a launch's size selects give the same
bits: a bunch in one launch against the same bunch in pieces that take other
register caps, for both solvers, with field-error harmonics, crossing capture
and space charge, and a host matrix through one range against two."""
import os
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

COLS = ("r", "vr", "z", "vz", "fi", "f5", "rf", "surv", "inj")
HARM = [{"m": 3, "amp_Gs": 2.0, "phase_deg": 10.0, "rmin": 7.0, "rmax": 10.0},
        {"m": 7, "amp_Gs": 1.0, "phase_deg": 50.0, "rmin": 8.0, "rmax": 8.2}]
_kept = {}


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("CUDA device required")


def machine(order, harm=False):
    from pyffa_b200 import synthetic
    from pyffa_b200.constants import FFAG_GlobalParameters
    from pyffa_b200.fields import FFAG_Bfield_analytical, FFAG_BField_Error, FFAG_EField_new
    if order not in _kept:
        cfg = synthetic.lattice_bmap(r_range=(7.9, 9.3, 0.01), theta_step_deg=0.1)
        stacks = synthetic.taylor_stacks(cfg, order) if order else None
        _kept[order] = FFAG_Bfield_analytical(config=cfg, max_order=order, stacks=stacks, AddNumricalMap=False)
    if "em" not in _kept:
        _kept["em"] = FFAG_EField_new(synthetic.emap_file(os.path.join(tempfile.mkdtemp(), "emap.txt")), EnableFlag=True)
    gp = FFAG_GlobalParameters()
    gp.AddBMap(_kept[order])
    gp.AddEMap(_kept["em"])
    if harm:
        gp.AddBHarmonics(FFAG_BField_Error(HARM, True))
    return gp


def rows(n, solver):
    from pyffa_b200 import synthetic
    from pyffa_b200.constants import FFAG_ConversionTools
    c = FFAG_ConversionTools()
    p = synthetic.gaussian_bunch(n, seed=9)
    p[:, 4] = np.random.default_rng(1).uniform(0.0, 2 * np.pi, n)
    v = c.ConvertPrzek2Vrzek_boris(p) if solver == "Boris" else c.ConvertPrzek2Vrzek(p)
    v[:, 7] = v[:, 8] = 1.0
    return v


def push(gp, v, solver, piece, sc=False, xing=False):
    from pyffa_b200 import synthetic
    from pyffa_b200.bunch import FFAG_Bunch
    from pyffa_b200.track import CrossingCapture, Pusher, StepClock
    n = v.shape[0]
    dt = synthetic.steps_per_turn_dt(steps_per_turn=720)
    b = FFAG_Bunch(v, BunchType=solver)
    for name in ("inj", "surv"):
        b.cols[name].fill_(1)
    if sc:
        g = torch.Generator(device="cuda")
        g.manual_seed(3)
        for name in ("e_pre_r", "e_pre_z", "e_pre_fi", "e_pp_r", "e_pp_z", "e_pp_fi"):
            b.cols[name].copy_(2e4 * torch.randn(n, dtype=torch.float64, device="cuda", generator=g))
        b.cols["sc_pre"].fill_(1)
        b.cols["sc_pp"].fill_(1)
    p = Pusher(b, gp, solver, "fp64", order=None)
    clock = StepClock(0.0, dt, gp.Emap, solver, b.device)
    clock.ensure(64)
    cap = CrossingCapture(b, [0.5], gp, dt) if xing else None
    x = cap.prepare(20) if xing else None
    for a in range(0, n, piece):
        p.push(clock, 12 if sc else 0, 20, 10 if sc else 0, xing=x, start=a, count=min(piece, n - a))
    torch.cuda.synchronize()
    out = {k: b.cols[k].clone() for k in COLS}
    if xing:
        r = cap.records()
        r[:, 1] = 0                      # the particle's place in its launch
        out["records"] = torch.from_numpy(r[np.lexsort(r.T)])
    return out


CASES = [("Boris", 2, {}), ("Boris", 3, {}), ("Boris", 1, {"harm": True}), ("Boris", 4, {"harm": True}),
         ("Boris", 2, {"xing": True}), ("Boris", 4, {"xing": True, "harm": True}), ("Boris", 2, {"sc": True}),
         ("Boris", 4, {"sc": True, "harm": True}), ("RK4", 2, {}), ("RK4", 4, {}), ("RK4", 3, {"sc": True}),
         ("RK4", 1, {"harm": True}), ("RK4", 2, {"xing": True})]


@pytest.mark.parametrize("solver,order,opt", CASES)
def test_pieces_equal_one_launch(solver, order, opt):
    """One launch of 22 and of 40 warps per SM against pieces of 6, 11 and 15."""
    opt = dict(opt)
    gp = machine(order, opt.pop("harm", False))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for warps in (22, 40):
        n = 32 * sms * warps - 5
        v = rows(n, solver)
        one = push(gp, v, solver, n, **opt)
        for piece in (6, 11, 15):
            got = push(gp, v, solver, 32 * sms * piece, **opt)
            for k in one:
                assert torch.equal(one[k], got[k]), (k, warps, piece)


@pytest.mark.parametrize("solver,order", [("Boris", 2), ("Boris", 4), ("RK4", 2)])
@pytest.mark.parametrize("n", [40_000, 75_000, 100_000])
def test_one_range_equals_two(solver, order, n):
    from pyffa_b200 import synthetic
    from pyffa_b200.track import MatrixTracker
    gp = machine(order)
    v = torch.from_numpy(rows(n, solver)).pin_memory()
    out = []
    for chunks in (1, 2):
        o = torch.empty_like(v).pin_memory()
        t = MatrixTracker(n, gp, solver, chunks=chunks)
        t.bind_clock(0.0, synthetic.steps_per_turn_dt(steps_per_turn=720), 32)
        t.run(v, o, 0, 32)
        torch.cuda.synchronize()
        out.append(o)
    assert torch.equal(out[0], out[1])
