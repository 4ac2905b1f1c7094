"""The near / far split's estimates lie within their bounds: every chain's estimate of the
field at its last point against the pair sum there, on planar emitters of 0.3 to 20 um with
electrons from 1e-6 nm above the cathode on, beside the supply nodes and anywhere, in both
precisions, and on a tip (near_bound.cu, linked with the library)."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_estimates_lie_within_their_bounds(rg, tmp_path):
    from rumdeed_gb300 import builder
    exe = str(tmp_path / "near_bound")
    subprocess.run([builder.nvcc(), *builder.ARCH, "-std=c++17", "-I", os.path.join(HERE, "..", "include"), "-o", exe,
                    os.path.join(HERE, "near_bound.cu"), "-L", builder.OUT_DIR, "-lrumdeed_gb300",
                    "-Xlinker", "-rpath=" + builder.OUT_DIR], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    print(r.stdout)
