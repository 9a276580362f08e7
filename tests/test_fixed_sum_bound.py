"""The node kernel's sum of eight forces in fixed point: the error bound that it
states, for sums whose large terms cancel too."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_the_stated_bound_holds_where_large_terms_cancel(tmp_path):
    nvcc = shutil.which(os.environ.get("NVCC", "nvcc"))
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "fixed_sum_bound_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", os.path.join(HERE, "fixed_sum_bound_check.cc"), "-o", exe], check=True,
                   capture_output=True)
    r = subprocess.run([exe, "50000"], capture_output=True, text=True, check=True)
    rows = [line.split() for line in r.stdout.splitlines()]
    assert len(rows) == 5
    for kind, fixed, fp64 in rows:
        assert float(fixed) <= 1.0, kind
    # additions in order are further off in general, and exact where pairs that
    # cancel follow one another
    by = {k: (float(a), float(b)) for k, a, b in rows}
    assert by["pairs_apart"][1] > 1.0 and by["nearly"][1] > 1.0 and by["alike"][1] > 1.0
