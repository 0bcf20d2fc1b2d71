"""The table that keeps the launcher's tensor maps (``csrc/recent_table.h``), on the CPU."""
import os
import subprocess

import pytest

from conftest import ROOT
from gcnasm_b200.build import _host_cxx

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("table") / "recent_table_check")
    subprocess.check_call([_host_cxx(), "-std=c++17", "-O1", "-g", "-pthread", "-I", os.path.join(ROOT, "gcnasm_b200", "csrc"),
                           os.path.join(HERE, "recent_table_check.cpp"), "-o", exe])
    return exe


@pytest.mark.parametrize("scenario", ["loop_is_kept", "oldest_go", "threads"])
def test_recent_table(program, scenario):
    r = subprocess.run([program, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.endswith("ok\n"), r.stdout + r.stderr
