"""The bounds-check build on the sweep solvers, the reference's V-cycles and the multigrid's masked
levels (tests/bounds_cases_sweeps.py, in a child process): no index check may fail, and every result
must equal the normal build's bit for bit."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from conftest import TESTS

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("CUDA device required", allow_module_level=True)


def _run(tmp_path, variant):
    out = str(tmp_path / f"{variant}.npz")
    env = dict(os.environ)
    env.pop("SG_LIBRARY_VARIANT", None)
    if variant == "bounds":
        env["SG_LIBRARY_VARIANT"] = "bounds"
    r = subprocess.run([sys.executable, os.path.join(TESTS, "bounds_cases_sweeps.py"), out], env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    return dict(np.load(out))


def test_index_checks_of_sweeps_pass_and_change_nothing(tmp_path):
    bc = _run(tmp_path, "bounds")
    assert int(bc["bounds_enabled"]) == 1
    assert int(bc["bounds_line"]) == 0, f"index check failed at line {int(bc['bounds_line'])} of unit " \
                                        f"{int(bc['bounds_unit'])}"
    ref = _run(tmp_path, "normal")
    assert int(ref["bounds_enabled"]) == 0
    for k in ref:
        if not k.startswith("bounds_"):
            assert np.array_equal(bc[k], ref[k], equal_nan=True), k
