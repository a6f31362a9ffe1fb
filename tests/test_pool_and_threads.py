"""Other Python threads run while the memory pool is busy: allocating and releasing a block give the interpreter up.

In a process of its own, on a library that stands in for the kernel library: every entry point succeeds, and the two of
the pool take 0.3 s."""
import os
import subprocess
import sys

from conftest import ROOT
from mytorch_b200.backends.cuda.env import _binding

PROGRAM = """
import threading, time
from mytorch_b200.backends.cuda.env import CudaEnv, CudaMemory
CudaEnv.instance()
for what in ("allocate", "destroy", "release"):
    block = CudaMemory(0, 64) if what != "allocate" else None
    stop, longest = threading.Event(), [0.0]
    def loader():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.002)
            now = time.perf_counter()
            longest[0], last = max(longest[0], now - last), now
    t = threading.Thread(target=loader)
    t.start()
    time.sleep(0.02)
    if what == "allocate":
        block = CudaMemory(0, 64)
    elif what == "destroy":
        block.destroy()
        assert block.ptr == 0
    else:
        del block
    stop.set()
    t.join()
    print(what, longest[0])
"""


def test_other_threads_run_while_the_pool_is_busy(tmp_path):
    slow = "usleep(300000);"
    source = ["#include <unistd.h>", 'extern "C" {', 'const char* mtb_last_error() { return ""; }',
              f"void* mtb_malloc(long long) {{ {slow} return (void*)0x1000; }}", f"int mtb_free(void*) {{ {slow} return 0; }}",
              "int mtb_device_count(int* n) { *n = 1; return 0; }", "int mtb_get_device(int* d) { *d = 0; return 0; }"]
    done = {"mtb_malloc", "mtb_free", "mtb_device_count", "mtb_get_device"}
    source += [f"long long {name}() {{ return 0; }}" for name in _binding.entry_points if name not in done] + ["}"]
    (tmp_path / "stand_in.cpp").write_text("\n".join(source))
    lib = tmp_path / "stand_in.so"
    subprocess.run(["g++", "-shared", "-fPIC", "-o", str(lib), str(tmp_path / "stand_in.cpp")], check=True)
    out = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, env={**os.environ, "MYTORCH_B200_LIB": str(lib)},
                         capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    gaps = dict(line.split() for line in out.stdout.split("\n") if line)
    assert set(gaps) == {"allocate", "destroy", "release"}
    for what, gap in gaps.items():
        assert float(gap) < 0.15, (what, gap)  # half of what the pool takes
