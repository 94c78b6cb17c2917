"""What a base conversion leaves for a transform stays within the bounds that the transform's double-precision butterflies start from."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_lazy_outputs_of_a_base_conversion(tmp_path):
    exe = str(tmp_path / "bconv_lazy_bounds")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-DCERIUM_EMU", "-I" + os.path.join(ROOT, "tests", "emu"),
                           "-I" + os.path.join(ROOT, "cerium_b200", "csrc"), "-o", exe, os.path.join(ROOT, "tests", "bconv_lazy_bounds.cpp"),
                           os.path.join(ROOT, "tests", "emu", "emu_runtime.cpp"), "-fopenmp"])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.startswith("OK"), out.stdout + out.stderr
