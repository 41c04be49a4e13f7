"""The real line operators' lane layout and block fragments, emulated on the
host for every line length against the dense circulant matrix."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_block_form_equals_the_dense_circulant(tmp_path):
    exe = str(tmp_path / "real_line_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "native", "real_line_check.cpp")])
    worst = float(subprocess.check_output([exe]))
    # values below 0.7, rows of nonnegative sum 1: at most N/4 + 4 roundings of
    # sums below 4 x 0.7 in a block, four blocks: (92 eps / 2) x 2.8 x 4 < 1.2e-13
    assert worst < 1.2e-13, worst
