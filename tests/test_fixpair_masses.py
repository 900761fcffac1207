"""The fixed-point terms with per-body masses on the host, against long double."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_light_partners_within_2_to_minus_55(tmp_path):
    """Partners down to 2^-84 of the heaviest body: an acceleration term and a potential term each
    within 2^-55 (0.25 units of 2^-53) of its own size, as with equal masses."""
    exe = tmp_path / "fixmass_check"
    subprocess.run(["g++", "-std=c++20", "-O2", "-ffp-contract=off",
                    f"-I{ROOT}/ode_prototyping_gb300/csrc",
                    os.path.join(ROOT, "tests", "cpp", "fixmass_check.cpp"), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out[2] == "ok" and float(out[0]) <= 0.25 and float(out[1]) <= 0.25, out
