"""Out of host memory at a C entry point: an error code and a message, no exception that leaves the library (which would end
the process). In a child process whose address space is closed and whose heap is used up."""
import subprocess
import sys
from pathlib import Path

import pytest

LIB = Path(__file__).resolve().parents[1] / "lokinfer_b200" / "liblkc.so"

CHILD = r"""
import ctypes, os, resource, sys
lib, libc = ctypes.CDLL(sys.argv[1]), ctypes.CDLL(None)
lib.lkc_last_error.restype = ctypes.c_char_p
malloc, free = libc.malloc, libc.free
malloc.restype, malloc.argtypes, free.argtypes = ctypes.c_void_p, [ctypes.c_size_t], [ctypes.c_void_p]

class Block(ctypes.Structure):
    _fields_ = [(n, ctypes.c_int64) for n in ("c", "k")] + [(n, ctypes.c_int64 * 6) for n in ("w", "b", "alpha", "state", "gb")]

class Io(ctypes.Structure):
    _fields_ = [(n, ctypes.c_int64) for n in ("x", "stats", "bank", "out", "out_stats", "l", "x_pitch", "out_pitch",
                                              "workspace", "workspace_bytes", "launches")]

blk, io, n, total = Block(c=16, k=3), Io(x=4096, bank=4096, out=4096, out_stats=4096, l=300, x_pitch=300, out_pitch=300), 4096, ctypes.c_int64()
for i in range(6):
    blk.w[i] = blk.b[i] = blk.alpha[i] = 4096
sizes, zeros, pins = (ctypes.c_int64 * n)(*[256] * n), (ctypes.c_int64 * n)(), (ctypes.c_int32 * n)()
offsets = (ctypes.c_int64 * n)()
calls = {"resblock": lambda: lib.lkc_resblock(ctypes.byref(blk), ctypes.byref(io), None),
         "plan_memory": lambda: lib.lkc_plan_memory(ctypes.c_int64(n), ctypes.c_int64(1), sizes, pins, zeros, zeros,
                                                    ctypes.c_int64(256), offsets, ctypes.byref(total))}
call = calls[sys.argv[2]]
assert call() == 0 and lib.lkc_last_error() == b""  # also touches the thread-local message
held = malloc(1 << 20)
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (used, resource.RLIM_INFINITY))
for size in [1 << 24, 1 << 20, 1 << 16, 1 << 14, 1 << 12] + list(range(2048, 0, -16)):
    while malloc(size):
        pass
rc = call()
free(held)
resource.setrlimit(resource.RLIMIT_AS, (resource.RLIM_INFINITY, resource.RLIM_INFINITY))
os.write(1, b"rc %d %s" % (rc, lib.lkc_last_error()))
os._exit(0)
"""


@pytest.mark.parametrize("entry", ["resblock", "plan_memory"])
def test_out_of_host_memory_is_an_error(entry):
    r = subprocess.run([sys.executable, "-c", CHILD, str(LIB), entry], capture_output=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stderr[-300:])
    assert r.stdout.startswith(b"rc 1 ") and b"out of host memory" in r.stdout, r.stdout
