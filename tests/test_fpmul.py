"""Products by a constant on the integer pipes, on the host, against the host's multiplication."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_products_bit_for_bit(tmp_path):
    exe = tmp_path / "fpmul_check"
    subprocess.run(["g++", "-std=c++20", "-O2", "-ffp-contract=off",
                    f"-I{ROOT}/ode_prototyping_gb300/csrc",
                    os.path.join(ROOT, "tests", "cpp", "fpmul_check.cpp"), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split()[-1] == "ok", out
