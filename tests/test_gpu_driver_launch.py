"""GPU: the line that the C++ drivers print ahead of a launch names the tile that is launched."""
import os
import subprocess

import pytest

from gcnasm_b200 import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,size,text", [
    ("gemm_a8w8_8wave", (256, 512, 1024), "tile_config=0, k_split=1, columns=32, sms="),
    ("gemm_a8w8_8wave", (333, 7168, 2048), "tile_config=0, k_split=1, columns=160, sms="),
    ("gemm_a8w8_8wave", (256, 8192, 1024), "tile_config=1, k_split=1, sms="),                 # 128 columns, the kind that tile 1 is
    ("gemm_a8w8_8wave", (256, 512, 8192), "tile_config=1, k_split=8, sms="),
    ("gemm_a8w8_8wave", (16, 512, 1024), "tile_config=3, k_split=1, sms="),
    ("gemm_a8w8_blockscale", (256, 512, 1024), "tile_config=0, k_split=1, columns=32, sms="),
    ("flatmm_a8w8", (256, 512, 1024), "tile_config=0, k_split=1, columns=32, sms="),
    ("gemm_a16w16", (256, 512, 512), "tile_config=0, k_split=1, columns=32, sms="),
    ("gemm_a16w16", (2000, 3000, 1024), "tile_config=0, k_split=1, columns=192, sms=")])
def test_the_printed_tile_is_the_launched_one(native, name, size, text):
    build.build_drivers()
    m, n, k = map(str, size)
    run = subprocess.run([os.path.join(build.BIN, name), "-m", m, "-n", n, "-k", k, "-b", "1", "-v", "0", "--warmup", "1", "--iters", "1"],
                         capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and text in run.stdout, run.stdout + run.stderr


def test_a_named_tile_is_printed(native):
    build.build_drivers()
    run = subprocess.run([os.path.join(build.BIN, "gemm_a8w8_8wave"), "-m", "256", "-n", "512", "-k", "1024", "-b", "1", "-v", "0", "--tile", "6", "--warmup", "1",
                          "--iters", "1"], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and "tile_config=6, k_split=1, sms=" in run.stdout
