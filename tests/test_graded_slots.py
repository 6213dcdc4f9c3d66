"""Which matrices a fixed-point field keeps in fp64 (fx_encode, fixed.cuh), on
the host: all whose small entries form a pattern, none of the generic ones, none
whose small entries are exact zeros. Either way the slot gives them back."""
import os
import subprocess

import pytest

from test_dfloat_products import INC, ROOT, _nvcc


@pytest.fixture(scope="module")
def counted(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("graded") / "graded_slots")
    src = os.path.join(ROOT, "tests", "native", "graded_slots.cu")
    try:
        r = subprocess.run([_nvcc(), "-O2", "-std=c++17", "-I", INC, src, "-o", exe], capture_output=True, text=True)
    except FileNotFoundError:
        pytest.skip("nvcc not available")
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout
    return {line.split()[0]: [int(v) for v in line.split()[1:]] for line in out.splitlines()}


@pytest.mark.parametrize("kind", ["weak", "diagonal", "su2", "real", "thin_row"])
def test_patterns_are_kept_in_fp64(counted, kind):
    n, graded, wrong = counted[kind]
    assert graded == n and wrong == 0


@pytest.mark.parametrize("kind", ["haar", "gaussian", "identity", "exact_su2"])
def test_generic_matrices_and_exact_zeros_are_not(counted, kind):
    n, graded, wrong = counted[kind]
    # eight of 18 numbers below 2^-7 of the norm by chance: under 1e-5 for
    # Gaussian entries (each 6%), and a small entry beside the zeros of an
    # embedded SU(2) matrix (8 numbers, each 1.2%) for one in ten
    assert graded <= {"gaussian": 1e-5, "exact_su2": 0.15}.get(kind, 0.0) * n
    assert wrong == 0


def test_results_below_the_normal_range(counted):
    assert counted["subnormal"][2] == 0
