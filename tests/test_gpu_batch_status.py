"""A batched solve whose applies report a wait that gave up fails, as rtg_solve does.  The report is a fake of the
library's own function, put in front of it in a child process: no wait on the GPU gives up."""
import os
import subprocess
import sys

import pytest

import golden_io  # noqa: F401  (puts the package on the path)
from rtg import build

pytestmark = pytest.mark.gpu

FAKE = r"""
#include "rtg_internal.h"
namespace rtg {
int apply_status(rtg_handle*, cudaStream_t) { return RTG_ERR_TIMEOUT; }
}
"""

CHILD = r"""
import sys
sys.path[:0] = %r
from rtg import _lib, workloads as W
from rtg.batch import BatchContext
ctx = BatchContext([W.batch_instance(k) for k in (1, 2)])
try:
    ctx.solve(ctx.forcing(), ctx.inflow(), rtol=1e-6)
except _lib.RtgError as e:
    assert "librtg error %%d:" %% _lib.RTG_ERR_TIMEOUT in str(e), e
    print("refused")
else:
    print("solved")
"""


@pytest.mark.parametrize("fake", [False, True])
def test_batched_solve_reads_the_status_of_its_applies(tmp_path, fake):
    env = dict(os.environ)
    if fake:
        src, lib = tmp_path / "fake.cpp", str(tmp_path / "fake.so")
        src.write_text(FAKE)
        r = subprocess.run([build.nvcc(), "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "--cudart", "none", "-I", build.INCLUDE, "-I", build.CSRC,
                            str(src), "-o", lib], capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        env["LD_PRELOAD"] = lib
    r = subprocess.run([sys.executable, "-c", CHILD % ([build.ROOT],)], capture_output=True, text=True, env=env, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split() == ["refused" if fake else "solved"]
