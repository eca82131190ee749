"""csrc/divide.h: the builder's division in integer and FP32 arithmetic gives
the bits of the FP64 division (every kept matrix element depends on them), on
operands of every exponent, next to powers of two, short ones, and quotients
next to midpoints, for any reciprocal estimate within 2^-21.  The device runs
the same source; the bit-exact builds of tests/test_gpu_build.py cover it."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_division_bits(tmp_path):
    exe = str(tmp_path / "divide_driver")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(HERE, "..", "adc_ottawa_gb300", "csrc"),
                    os.path.join(HERE, "host", "divide_driver.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe, "30000000"], capture_output=True, text=True, check=True)
    assert out.stdout.strip() == "0"
