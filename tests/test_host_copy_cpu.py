"""The threads that share copies of pageable operands, without a GPU: the bytes are right, the
threads take no signals, and a program may close the library while they live."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
import _ctypes, ctypes, os, sys, time
def tasks():
    return set(os.listdir("/proc/self/task"))
lib = ctypes.CDLL(sys.argv[1])
copy = lib.probe_copy
copy.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_size_t, ctypes.c_size_t]
before = tasks()
for width, rows, pitch in ((1 << 20, 1, 1 << 20), (4099, 200, 5000), (100, 10, 100), (1000, 1000, 1000)):
    src = os.urandom(pitch * rows)
    dst = ctypes.create_string_buffer(width * rows)
    for _ in range(20):
        copy(dst, src, width, rows, pitch)
    assert dst.raw == b"".join(src[r * pitch:r * pitch + width] for r in range(rows))
helpers = tasks() - before
for t in helpers:
    blocked = int(next(l for l in open(f"/proc/self/task/{t}/status") if l.startswith("SigBlk")).split()[1], 16)
    for sig in (1, 2, 10, 14, 15, 17):
        assert blocked >> (sig - 1) & 1, ("a helper thread takes signal", sig)
own = int(next(l for l in open("/proc/self/status") if l.startswith("SigBlk")).split()[1], 16)
assert own == 0, "the caller's signal mask was left changed"
copy(dst, src, width, rows, pitch)
_ctypes.dlclose(lib._handle)   # the helpers still watch for the next copy
time.sleep(0.05)
print("helpers", len(helpers))
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    out = tmp_path_factory.mktemp("host_copy") / "libprobe.so"
    subprocess.run(["nvcc", "-std=c++17", "-O2", "-shared", "-Xcompiler", "-fPIC,-fvisibility=default", "-x", "c++",
                    "-o", str(out), str(ROOT / "tests" / "cpp" / "host_copy_probe.cc"), "-lcudart", "-ldl"], check=True)
    return out


def test_threads_keep_to_themselves(probe):
    done = subprocess.run([sys.executable, "-c", PROGRAM, str(probe)], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stderr
    word, helpers = done.stdout.split()
    # (whether the C++ library counts the machine's cores or the process's differs)
    fewest = min(len(os.sched_getaffinity(0)), os.cpu_count() or 1)
    assert word == "helpers" and (1 if fewest >= 4 else 0) <= int(helpers) <= 3
