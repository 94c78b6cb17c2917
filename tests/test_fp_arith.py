"""Device arithmetic checked on the CPU against 128-bit integers: programs that include the library's own kernel headers are
compiled and run.  tests/fp_arith_check.cpp: the double-precision modular arithmetic of the transforms (primes below 2^50).
tests/bconv_finish_check.cpp: the last step of a base conversion."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fp_mulmod_reduce_and_conversions_are_exact(tmp_path):
    exe = str(tmp_path / "fp_arith_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-DCERIUM_EMU",
                           "-I" + os.path.join(ROOT, "tests", "emu"), "-I" + os.path.join(ROOT, "cerium_b200", "csrc"),
                           "-o", exe, os.path.join(ROOT, "tests", "fp_arith_check.cpp")])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.startswith("OK"), out.stdout + out.stderr
    worst = float(out.stdout.split()[1])
    assert worst <= 0.5 + 4.0 / 32.0 + 1e-6   # |y| <= 4q


def test_bconv_finish_is_exact_up_to_the_largest_sum(tmp_path):
    exe = str(tmp_path / "bconv_finish_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-DCERIUM_EMU", "-I" + os.path.join(ROOT, "tests", "emu"),
                           "-I" + os.path.join(ROOT, "cerium_b200", "csrc"), "-o", exe,
                           os.path.join(ROOT, "tests", "bconv_finish_check.cpp"), os.path.join(ROOT, "tests", "emu", "emu_runtime.cpp"),
                           "-fopenmp"])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.startswith("OK"), out.stdout + out.stderr
