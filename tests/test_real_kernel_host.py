"""The circulant kernels that the line operators are made of, for every line length."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_kernels_equal_the_plain_sums(tmp_path):
    exe = str(tmp_path / "real_kernel_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "native", "real_kernel_check.cpp")])
    assert int(subprocess.check_output([exe])) == 0   # the same terms in the same order
