"""The bounds-checked build on what test_gpu_checked's selection does not reach:
waves with and without a hand-over, the batch's path-slot pool, caller BVHs that
share subtrees or reach the stack's bound, and the adjoint."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
pytestmark = pytest.mark.gpu


def test_forms_pass_with_bounds_checks():
    from raymotion_b200 import build
    if not build.LIB_CHECKED.exists():
        build.build(checked=True)
    env = dict(os.environ, RAYMOTION_CUDA_CHECKED="1")
    sel = ("waves_match_the_oracle or pool_tunings or large_sample_counts_equal_the_oracle or shared_subtrees or "
           "most_subtrees_pending or collapse_forms or clamped_channels or more_materials or equal_terms")
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-p", "no:cacheprovider", "-m", "gpu", "-k", sel,
                        "tests/test_gpu_forms.py", "tests/test_gpu_caller_bvh.py", "tests/test_gpu_uploads.py",
                        "tests/test_gpu_adjoint_tasks.py", "tests/test_gpu_adjoint_sums.py"],
                       capture_output=True, text=True, env=env, cwd=ROOT, timeout=1800)
    assert r.returncode == 0, r.stdout[-4000:] + r.stderr[-2000:]
    assert " passed" in r.stdout and "failed" not in r.stdout
