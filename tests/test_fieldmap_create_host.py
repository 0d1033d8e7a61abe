"""ffa_fieldmap_create on the host: its errors come back as codes, and a
mid-plane map (no node tables) can be made without a device."""
import subprocess
import sys

import pytest

from pyffa_b200 import build

CODE = """
import ctypes, resource, sys
from pyffa_b200 import _lib
L = ctypes.CDLL(sys.argv[1])
d = _lib.FieldDesc()
d.nsectors, d.n_convex, d.max_order, d.B0, d.k = 12, 1, 0, 1.0, 7.6
d.convex[:5] = [0.1, 0.2, float(sys.argv[2]), 1.0, 1.0]
d.r_min, d.r_step, d.r_size = 8.0, 0.001, 1301
if int(sys.argv[3]):
    pages = int(open("/proc/self/statm").read().split()[0])
    resource.setrlimit(resource.RLIMIT_AS, (pages * resource.getpagesize() + int(sys.argv[3]),) * 2)
h = ctypes.c_void_p()
print(L.ffa_fieldmap_create(ctypes.byref(d), None, ctypes.byref(h)), int(bool(h)))
"""


def create(fringe, room=0):
    """(return code, whether a map came back) of a mid-plane map's creation in
    a process of its own that may map `room` more bytes (0: no limit)."""
    r = subprocess.run([sys.executable, "-c", CODE, build.build(), str(fringe), str(room)], capture_output=True,
                       text=True, cwd=build.REPO_DIR)
    assert r.returncode == 0, (r.returncode, r.stderr[-500:])
    return tuple(int(x) for x in r.stdout.split())


def test_no_room_for_the_tables_is_an_error_code():
    # a sharp fringe's flutter table takes 4.4 MB; the process has 2 MB left
    assert create(0.0035, 2 << 20) == (3, 0)          # FFA_ERR_NOMEM


def test_mid_plane_map_without_a_device():
    torch = pytest.importorskip("torch")
    if torch.cuda.is_available():
        pytest.skip("there is a device")
    assert create(0.19) == (0, 1)
    assert create(0.0035) == (0, 1)
