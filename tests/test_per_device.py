"""Launch limits kept per device (pb::PerDevice in prism_b200/csrc/common.h), checked on the host:
tests/cpp/per_device_check.cpp compiles the header against a fake cudaGetDevice. Every cluster
limit of the kernels is kept by it."""
import glob
import os
import re
import shutil
import subprocess

import pytest

from tests.test_arena import ROOT, _cuda_include


def test_per_device_logic(tmp_path):
    inc = _cuda_include()
    if inc is None or shutil.which("g++") is None:
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path / "per_device_check")
    src = os.path.join(ROOT, "tests", "cpp", "per_device_check.cpp")
    subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", "-I", inc, src, "-o", exe], check=True,
                   capture_output=True, text=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stderr


def test_cluster_limits_are_kept_per_device():
    """cudaFuncSetAttribute and cluster occupancy concern the current device: a static result of
    theirs has to be a PerDevice."""
    uses = 0
    for path in glob.glob(os.path.join(ROOT, "prism_b200", "csrc", "*.cu")):
        text = open(path).read()
        assert "NonPortableClusterSizeAllowed" not in text, path  # clusterPlaced sets it
        assert not re.search(r"static (const )?int \w+ = (\[\] \{[^}]*)?clusterPlaced", text), path
        uses += len(re.findall(r"static PerDevice \w+;\s+return \w+\.get\(\[\] \{\s*(return )?clusterPlaced", text))
    assert uses == 3
