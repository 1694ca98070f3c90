"""The suites of the newer kernels on the bounds-checked build (see test_gpu_bounds_check.py):
uneven tiles, the FP64 tensor-core tiles, long tile lists, sparse and far blobs, the packed
transforms, the small GMRES and the batches on unpacked grids.  Their timing tests stay out:
the checks cost time.  And, on the CPU, that every source with a bounds record has checks
to fill it."""
import glob
import os
import re
import subprocess
import sys

import pytest

from timstochrigidbodiessim_b200 import capi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SUITES = ["tests/test_gpu_uneven_tiles.py", "tests/test_gpu_tensor_tiles_fp64.py", "tests/test_gpu_long_tile_lists.py",
          "tests/test_gpu_sparse_interpolation.py", "tests/test_gpu_sparse_uneven.py", "tests/test_gpu_far_positions.py", "tests/test_gpu_packed_solve.py",
          "tests/test_gpu_slender_noise.py", "tests/test_gpu_small_gmres.py", "tests/test_gpu_gmres_columns.py", "tests/test_gpu_batch_unpacked.py"]


def test_sources_with_a_bounds_record_check_something():
    seen = 0
    for path in glob.glob(os.path.join(ROOT, "timstochrigidbodiessim_b200", "csrc", "*.cu")):
        text = open(path).read()
        if not re.search(r"^FCM_BOUNDS_READER\(", text, re.M):
            continue
        seen += 1
        for kernel in re.split(r"__global__", text)[1:]:
            name = re.search(r"\b(k_packed_\w+)\(", kernel)
            if name and name.group(1) in ("k_packed_z", "k_packed_y", "k_packed_plane"):
                assert "FCM_INB(" in kernel, name.group(1)
        assert "FCM_INB(" in text, os.path.basename(path)
    assert seen >= 5


@pytest.mark.gpu
def test_suites_on_bounds_checked_build(gpu):
    if os.environ.get("FCM_B200_BOUNDS_CHECK") == "1":
        pytest.skip("already running on the bounds-checked build")
    assert os.path.exists(capi.DEBUG_LIB_PATH), "libfcm_b200_debug.so not built (python -m timstochrigidbodiessim_b200.build)"
    env = dict(os.environ, FCM_B200_BOUNDS_CHECK="1")
    r = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-m", "gpu", "-p", "no:cacheprovider", "-k",
                        "not time"] + SUITES, cwd=ROOT, env=env, capture_output=True, text=True, timeout=1800)
    tail = (r.stdout + r.stderr)[-3000:]
    assert r.returncode == 0, tail
    assert " passed" in r.stdout and " failed" not in r.stdout, tail
