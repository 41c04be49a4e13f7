"""The circulant kernels that the line operators are made of, for every line length."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_kernels_equal_the_plain_sums(tmp_path):
    exe = str(tmp_path / "real_kernel_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "native", "real_kernel_check.cpp")])
    # an entry of c is a mean of N <= 352 terms of at most one, three roundings of 2^-64
    # each: 3 x 352 x 2^-64 < 5.8e-17; T is a sum of two, on either side
    assert float(subprocess.check_output([exe])) < 2.4e-16
