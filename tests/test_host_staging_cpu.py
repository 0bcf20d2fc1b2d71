"""The pinned ring and the copy threads of the host-buffer entry (``csrc/host_staging.h``), compiled against a stand-in for the
CUDA runtime in which copies run late and single calls fail."""
import os
import subprocess

import pytest

from conftest import ROOT
from gcnasm_b200.build import _host_cxx

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("staging") / "host_staging_check")
    subprocess.check_call([_host_cxx(), "-std=c++17", "-O1", "-g", "-pthread", "-I", os.path.join(HERE, "fake_cuda"),
                           "-I", os.path.join(ROOT, "gcnasm_b200", "csrc"), os.path.join(HERE, "host_staging_check.cpp"), "-o", exe])
    return exe


@pytest.mark.parametrize("scenario", ["round_trip", "failed_call", "no_ring", "no_memory"])
def test_host_staging(program, scenario):
    r = subprocess.run([program, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.endswith("ok\n"), r.stdout + r.stderr
