"""After a bounded wait of the jumps gave up, the next step starts from clean counters
(near_reset): the set-up launches zero what an unfinished jump had counted (near_reset.cu,
linked with the library)."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_counters_are_zero_before_the_first_jump(rg, tmp_path):
    from rumdeed_gb300 import builder
    exe = str(tmp_path / "near_reset")
    subprocess.run([builder.nvcc(), *builder.ARCH, "-std=c++17", "-I", os.path.join(HERE, "..", "include"), "-o", exe,
                    os.path.join(HERE, "near_reset.cu"), "-L", builder.OUT_DIR, "-lrumdeed_gb300",
                    "-Xlinker", "-rpath=" + builder.OUT_DIR], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
