"""The fixed-point pair term on the host, against long double."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_terms_within_2_to_minus_55(tmp_path):
    """Separations over the whole window, systems far from the origin, with and without softening:
    every term within 2^-55 (0.25 units of 2^-53) of its size.  The seed's error in
    the host's rsqrt stays inside the SFU's bound, so the same integers follow."""
    exe = tmp_path / "fixpair_check"
    subprocess.run(["g++", "-std=c++20", "-O2", "-ffp-contract=off",
                    f"-I{ROOT}/ode_prototyping_gb300/csrc",
                    os.path.join(ROOT, "tests", "cpp", "fixpair_check.cpp"), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out[2] == "ok" and float(out[1]) <= 0.25, out
