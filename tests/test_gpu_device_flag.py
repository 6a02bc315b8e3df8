"""Device error flags that an asynchronous call leaves are kept for the next blocking one
(tests/cpp/device_flag.cu; no wait runs out here: the flag is set from the host)."""
import os
import subprocess

import pytest

from simdgraphprocessing_gb300 import build as B

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_flags_outlive_asynchronous_calls(eh, tmp_path):
    exe, libdir = str(tmp_path / "device_flag"), os.path.dirname(eh.lib_path())
    cmd = [B._nvcc(), *B.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", B.CSRC, "-I", B.INCLUDE,
           os.path.join(ROOT, "tests", "cpp", "device_flag.cu"), "-o", exe, "-L", libdir, "-leh_gb300",
           "-Xlinker", "-rpath," + libdir]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert r.returncode == 0, r.stdout[-3000:]
    r = subprocess.run([exe], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout[-3000:]
