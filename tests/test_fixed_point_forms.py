"""Host checks of the fixed-point line operations (csrc/igr_fix.cuh) in the
forms that the kernels use; tests/fixed_point_forms.cpp says what each holds."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fix") / "fixed_point_forms")
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", out, os.path.join(HERE, "fixed_point_forms.cpp")], check=True)
    return out


@pytest.mark.parametrize("name", ["flux_range", "mean", "odd", "face_sides", "leading", "forms", "nonfinite"])
def test_form(exe, name):
    r = subprocess.run([exe, name], capture_output=True, text=True)
    bad = [ln for ln in r.stdout.splitlines() if " ok " not in ln]
    assert r.returncode == 0 and not bad, "\n".join(bad[:20]) or r.stderr
