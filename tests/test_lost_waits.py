"""A block whose wait for another block runs out (made to in the bounds-check build, which gives the
wait up at once): no finite value depends on it, solves to a tolerance raise instead of reporting
convergence, the wait is counted, and the next solve is right (tests/lost_waits.py, in a child
process)."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from conftest import TESTS, package

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("CUDA device required", allow_module_level=True)

sg = package()


@pytest.fixture(scope="module")
def runs(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("waits") / "out.npz")
    r = subprocess.run([sys.executable, os.path.join(TESTS, "lost_waits.py"), out],
                       env=dict(os.environ, SG_LIBRARY_VARIANT="bounds"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    return dict(np.load(out))


@pytest.mark.parametrize("name", ["jacobi", "sor", "sor_one_trade", "gauss_seidel", "vcycles", "tolerance", "mixed"])
def test_nothing_finite_depends_on_a_lost_wait(runs, name):
    before, lost, after = (runs[f"{name}_{r}"] for r in ("before", "lost", "after"))
    assert np.isfinite(before).all() and np.array_equal(before, after)
    assert int(runs[f"{name}_before_count"]) == 0 and int(runs[f"{name}_after_count"]) == 0
    assert int(runs[f"{name}_lost_count"]) > 0
    if name in ("tolerance", "mixed"):
        assert "non-finite" in str(runs[f"{name}_lost_raised"])
    else:
        assert np.isnan(lost).any() and np.all(np.isnan(lost) | (lost == before))
    assert str(runs[f"{name}_before_raised"]) == "" == str(runs[f"{name}_after_raised"])


def test_normal_build_counts_none():
    assert sg._lib.lost_waits() == 0
    assert sg._lib.load().sg_bounds_lose_waits(1) == sg._lib.SG_ERR_ARG
