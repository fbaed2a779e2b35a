"""Creating a handle while the host runs out of memory: whichever of its large allocations
fails, the call returns an error (nothing leaves the C entry), and the next call succeeds."""
import os
import shutil
import subprocess
import sys

import pytest

from storm_b200 import fvt

pytestmark = pytest.mark.gpu

# operator new that refuses the k-th request of 16 KB or more since arm(k)
HOOK = r"""
#include <cstdlib>
#include <new>
static int left = 0, seen = 0;
extern "C" void arm(int k) { left = k; seen = 0; }
extern "C" int large(void) { return seen; }
void* operator new(std::size_t n) {
  if (left > 0 && n >= 16384 && ++seen == left) throw std::bad_alloc();
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
"""
CHILD = r"""
import ctypes, sys
from storm_b200 import abi, fvt, scenarios
hook = ctypes.CDLL(sys.argv[1])
sc = scenarios.channel(nx=80, ny=20)
sc.options.precision = int(sys.argv[2])
pm = fvt.build_mesh(sc.problem)
fvt.Solver(pm, sc.options, keep=pm).close()
k = 0
while True:
    k += 1
    hook.arm(k)
    try:
        s = fvt.Solver(pm, sc.options, keep=pm)
    except fvt.StormError as e:
        hook.arm(0)
        assert e.code == abi.STORM_ERR_NOMEM, e
        continue
    n = hook.large()
    hook.arm(0)
    s.set_state(sc.h0, sc.u0, sc.v0)
    s.step(2)
    s.close()
    if n < k:  # no request was refused
        break
print("refused", k - 1)
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="compiles its hook: needs g++")
@pytest.mark.parametrize("precision", [0, 1])
def test_every_large_allocation(precision, tmp_path, storm_lib):
    (tmp_path / "hook.cpp").write_text(HOOK)
    so = str(tmp_path / "hook.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-o", so, str(tmp_path / "hook.cpp")], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(fvt.__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD, so, str(precision)], cwd=root, timeout=300, text=True,
                       capture_output=True, env={**os.environ, "LD_PRELOAD": so})
    assert r.returncode == 0, r.stderr[-2000:]
    assert int(r.stdout.split()[-1]) > 100
