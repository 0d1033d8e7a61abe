"""A mid-plane map made while a stream is captured works as one made before,
and the capture goes on."""
import ctypes
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("CUDA device required")


def test_mid_plane_map_during_capture():
    from pyffa_b200 import _lib, seo, synthetic
    from pyffa_b200.constants import FFAG_ConversionTools, Q
    from pyffa_b200.fields import FFAG_Bfield_analytical
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        bm = FFAG_Bfield_analytical(config=synthetic.lattice_bmap(), max_order=0, AddNumricalMap=False)
    x0 = np.array([[8.13, 0.1168, 1e-3, 0.0, FFAG_ConversionTools().Ek2P(300.0)]])
    want = seo.ThetaTracker(bm, Q).run(x0, 2 * np.pi / 12, 0.001, 0, False)[0]
    h, d = ctypes.c_void_p(), bm.field_desc()
    x = torch.zeros(4, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x += 1
        rc = _lib.lib().ffa_fieldmap_create(ctypes.byref(d), torch.cuda.current_stream().cuda_stream, ctypes.byref(h))
        x += 1
    assert rc == 0
    g.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 4
    t = seo.ThetaTracker(bm, Q)
    t.fm = type("Map", (), {"handle": h})()
    assert np.array_equal(t.run(x0, 2 * np.pi / 12, 0.001, 0, False)[0], want)
    assert _lib.lib().ffa_fieldmap_destroy(h) == 0
