"""A host that refuses page-locked memory: the same calls, the same bits.  The
host side of the engine is compiled here with cudaHostAlloc replaced by a
refusal and linked to the library's kernels; a child process runs it."""
import importlib
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

SHIM = """#pragma once
#include <cuda_runtime.h>
#include <atomic>
inline std::atomic<int> refusals{0};
inline cudaError_t refuse_host_alloc(void** p, size_t, unsigned) {
    *p = nullptr;
    ++refusals;
    return cudaErrorMemoryAllocation;
}
extern "C" int refused_allocations() { return refusals.load(); }
#define cudaHostAlloc refuse_host_alloc
"""

RUN = """
import ctypes, importlib, sys
from pathlib import Path
import numpy as np
sys.path.insert(0, {root!r})
cfsb = importlib.import_module("2d_compressible_flow_solver_b200")
wl = importlib.import_module("2d_compressible_flow_solver_b200.workloads")
if {lib!r}:
    cfsb.LIB_PATH = Path({lib!r})
out = {{}}
for prec in (0, 1, 2):
    for nx, ny in ((48, 40), (300, 200)):
        U = wl.riemann_quadrants(nx, ny, seed=5).U0
        with cfsb.Solver(nx, ny, precision=prec, rk=cfsb.RK_TVD3_REFERENCE) as s:
            s.set_state(U)
            dt = s.compute_dt(0.4)
            s.step(dt)
            t, last = s.advance(3, cfl=0.4)
            s.steps_begin(cfl=0.4)
            for _ in range(3):
                s.steps_stage()
            t2, _ = s.steps_end()
            s.synchronize()
            again = s.compute_dt(0.4)
            out[f"{{prec}}_{{nx}}"] = s.get_state()
            out[f"t{{prec}}_{{nx}}"] = np.array([dt, t, last, t2, again])
if {lib!r}:
    assert ctypes.CDLL({lib!r}).refused_allocations() >= 6
np.savez({out!r}, **out)
"""


def test_results_come_through_device_memory(cfsb, tmp_path):
    build = importlib.import_module("2d_compressible_flow_solver_b200.build")
    (tmp_path / "refuse.h").write_text(SHIM)
    lib = tmp_path / "libcfs_refused.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", "-include", str(tmp_path / "refuse.h"),
                    f"-I{build.CSRC}", f"-I{build.INCLUDE}", f"-I{build.CUDA_HOME / 'include'}",
                    str(build.CSRC / "cfs_api.cpp"), "-o", str(lib), str(build.LIB), f"-Wl,-rpath,{build.LIB.parent}",
                    "-Wl,-Bsymbolic", f"-L{build.CUDA_HOME / 'lib64'}", "-lcudart_static", "-lrt", "-ldl"], check=True)
    got = {}
    for name, path in (("plain", ""), ("refused", str(lib))):
        npz = tmp_path / f"{name}.npz"
        r = subprocess.run([sys.executable, "-c", RUN.format(root=str(ROOT), lib=path, out=str(npz))],
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        got[name] = dict(np.load(npz))
    for k, v in got["plain"].items():
        assert np.all(np.isfinite(v)) and np.array_equal(v, got["refused"][k]), k
