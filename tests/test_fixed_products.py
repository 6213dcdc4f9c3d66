"""Accuracy of the block fixed-point row products (fixed.cuh), measured on the
host: device and host forms are the same source. Chains of two products
against long double, beside the same chains in fp64.

The bound: an operand holds 60 fraction bits of its norm and a row product
drops less than 2^-59 of it (the low x low limbs and the final shift), so a
chain of two stays within a few 2^-58, under fp64's 2^-53 per rounding. For
general matrices the exponent comes from an upper bound of the spectral norm
(at most 6 times it), which costs up to 2.6 bits per factor."""
import os
import subprocess

import pytest

from test_dfloat_products import INC, ROOT, _nvcc

SRC = os.path.join(ROOT, "tests", "native", "fixed_products.cu")


@pytest.fixture(scope="module")
def measured(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fxp") / "fixed_products")
    try:
        r = subprocess.run([_nvcc(), "-O2", "-std=c++17", "-I", INC, SRC, "-o", exe], capture_output=True, text=True)
    except FileNotFoundError:
        pytest.skip("nvcc not available")
    assert r.returncode == 0, "host build of the product check failed:\n" + r.stdout + r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout
    print(out)
    return {line.split()[0]: [float(v) for v in line.split()[1:]] for line in out.splitlines()}


@pytest.mark.parametrize("kind", ["unitary", "gaussian", "graded"])
def test_chain_is_no_further_off_than_fp64(measured, kind):
    rms, worst, rms64, worst64, conversion, shifted = measured[kind]
    assert rms <= rms64 and worst <= worst64
    assert worst <= 2.0 ** -53 and conversion <= 2.0 ** -53
    assert shifted == 0  # unitary matrices have exponent 0


def test_special_values(measured):
    assert measured["special"] == [0]
