"""Host allocations that fail inside a C entry are an error code, not an abort of the
process: a child with a limited address space asks for a sum of 2^31 - 1 terms."""
import subprocess
import sys

CHILD = """
import ctypes, resource, sys
sys.path.insert(0, {root!r})
from qaravan_gb300 import _lib
L = _lib.lib()
buf = ctypes.create_string_buffer(64)
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (used + (1 << 30), used + (1 << 30)))
at = ctypes.addressof(buf)
rc = [f(at, 1, 2, b"ii", None, 2 ** 31 - 1, 1, 0, at, at, 2 ** 62, None)
      for f in (L.qgb_pauli_expectation, L.qgb_dm_pauli_expectation)]
print(rc, L.qgb_last_error().decode())
"""


def test_no_memory_for_the_terms():
    from qaravan_gb300 import _lib, build
    build.build()
    import os
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=root)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-500:]
    assert r.stdout.strip() == f"[{_lib.QGB_EINVAL}, {_lib.QGB_EINVAL}] out of host memory"
