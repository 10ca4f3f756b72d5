"""A power spectrum with more annuli than the caller has room for is refused before anything
is listed or allocated, however many they are (no GPU: refused on the host).  In a child
process with little address space, where listing them first would abort the process."""
import subprocess
import sys

import pytest

CHILD = r"""
import ctypes as C, resource, sys
from trophic_maelstorm_gb300 import _lib
L = _lib.lib()
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (used + (512 << 20),) * 2)
kv, pw, nb = (C.c_double * 16)(), (C.c_double * 16)(), C.c_int(-1)
side, width, room = int(sys.argv[1]), float(sys.argv[2]), int(sys.argv[3])
field = (C.c_double * 16)()                       # never read
rc = L.tm_power_spectrum_device(C.cast(field, C.c_void_p), 0, side, width, None, C.cast(kv, C.POINTER(C.c_double)),
                                C.cast(pw, C.POINTER(C.c_double)), room, C.byref(nb))
print(rc, nb.value)
"""


@pytest.mark.parametrize("side,width,room,bins", [(64, 1e-12, 16, 2147483647), (64, 1e-300, 16, 2147483647),
                                                  (46340, 1e-4, 16, 231700000), (64, 0.5, 16, 64), (32, 1.0, 0, 16)])
def test_too_many_annuli_are_refused(side, width, room, bins):
    r = subprocess.run([sys.executable, "-c", CHILD, str(side), repr(width), str(room)], capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0, r.stderr[-400:]
    rc, nb = (int(x) for x in r.stdout.split())
    assert rc == -1 and abs(nb - bins) <= 1
