"""The fixed-point line contractions of csrc/igr_fix.cuh, built for the host,
against long double sums: every form (rows, columns, scaled, with accumulands),
p = 1..4, at the ends of the integer path's range and beyond it."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_line_contractions_on_the_host(tmp_path):
    exe = str(tmp_path / "fixed_point_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", exe, os.path.join(HERE, "fixed_point_check.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    bad = [ln for ln in r.stdout.splitlines() if " ok " not in ln]
    assert r.returncode == 0 and not bad, "\n".join(bad[:20])
