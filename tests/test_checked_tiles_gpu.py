"""The tiled step group's suites, and the raster sort's, with the index-checking
library (see test_checked_build_gpu.py): every index that the kernels read from
memory is tested before use, and no test fires."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SUITES = ["tests/test_tile_group_gpu.py", "tests/test_tile_stdp_gpu.py", "tests/test_tile_lists_gpu.py",
          "tests/test_tile_timeout_gpu.py", "tests/test_tile_epochs_gpu.py", "tests/test_step_form_gpu.py",
          "tests/test_raster_sort_gpu.py"]


@pytest.mark.gpu
def test_tile_suites_pass_with_index_checks():
    lib = os.path.join(ROOT, "mgbrain_b200", "lib", "libmgbrain_b200_checked.so")
    assert os.path.exists(lib), "build the checked library (python -m mgbrain_b200.build --checked)"
    env = dict(os.environ, MGBRAIN_LIB="checked")
    r = subprocess.run([sys.executable, "-c", "import mgbrain_b200 as m; print(m.capi.LIB_PATH)"], env=env, cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.stdout.strip().endswith("libmgbrain_b200_checked.so"), r.stdout + r.stderr
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider"] + SUITES,
                       env=env, cwd=ROOT, capture_output=True, text=True, timeout=1800)
    assert r.returncode == 0, r.stdout[-4000:]
