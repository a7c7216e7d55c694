"""The host's parallel loops where no thread can be started (the address space is used up, so a
thread's stack cannot be mapped): the calling thread takes the chunks itself. And where an
iteration throws, in the calling thread's chunk or another's: the caller gets the exception. Each
in a process of its own, which the library must not end."""
import subprocess
import sys

import pytest

CHILD = """
import ctypes as C, resource, sys
L = C.CDLL({so!r})
L.gpl_rules_parallel_sum.restype = C.c_int64
L.gpl_rules_parallel_sum.argtypes = [C.c_int64, C.c_int64]
if {starved}:
    used = int(open('/proc/self/statm').read().split()[0]) * resource.getpagesize()
    resource.setrlimit(resource.RLIMIT_AS, (used + (1 << 20), resource.RLIM_INFINITY))
print(L.gpl_rules_parallel_sum({n}, {stop}))
"""


@pytest.mark.parametrize("starved", [False, True])
@pytest.mark.parametrize("n,stop,want", [(0, -1, 0), (1, -1, 0), (1000, -1, 499500), (1000, 0, -1), (1000, 999, -1), (1000, 500, -1)])
def test_parallel_loop(starved, n, stop, want):
    from gpl_b200 import build
    code = CHILD.format(so=build.build(), starved=starved, n=n, stop=stop)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    assert int(r.stdout) == want
