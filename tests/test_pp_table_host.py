"""The FP64 pair table on the host: which interval count parameters take, and
that psi and g are within the table's limit of themselves everywhere on [0, rc],
against the closed form in extended precision. The counts are those the GPU
tests of the pair loop rely on.

Tolerance: the builder holds 4e-16 at the ends and the middle of every interval,
where an interpolant through Chebyshev points and its slope are worst; a tenth
more for the points between.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

#: (kappa, alpha, rc) -> intervals
COUNTS = {
    # test_gpu_batch_fp64.py
    (0.1, 0.46, 2.975): 128, (0.0, 0.9, 2.975): 256, (6.0, 0.85, 2.975): 512, (40.0, 1.5, 2.975): 0,
    # test_gpu_pp_table.py, with the four above
    (1.0, 0.6, 2.975): 128, (3.0, 0.45, 2.975): 256,
    # test_gpu_pp_pair.py
    (0.5, 0.72, 5.0): 512, (2.0, 0.72, 4.9): 512, (0.0, 0.75, 4.8): 512, (3.0, 0.65, 5.1): 512,
    (1.0, 0.3, 3.3): 128, (9.0, 0.6, 5.3): 1024,
    # runs of production size
    (2.0, 0.6, 6.0): 512, (0.1, 0.46, 7.8): 512, (1.0, 0.5, 7.0): 512, (3.0, 0.2, 20.0): 1024,
}


@pytest.fixture(scope="module")
def results(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path_factory.mktemp("pp") / "check")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "md-force-routines_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "pp_table_check.cpp")], check=True)
    args = [repr(v) for p in COUNTS for v in p]
    out = subprocess.run([exe, *args], capture_output=True, text=True, timeout=120, check=True).stdout
    return dict(zip(COUNTS, (line.split() for line in out.splitlines())))


@pytest.mark.parametrize("param", COUNTS)
def test_interval_count_and_error(results, param):
    n, epsi, eg = results[param]
    assert int(n) == COUNTS[param]
    assert float(epsi) <= 4.4e-16 and float(eg) <= 4.4e-16
