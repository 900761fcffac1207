"""Small components of the fixed-point acceleration terms on the host, against long double."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_components_within_2_to_minus_53(tmp_path):
    """Every component of a term above 2^-26 of the term, and not the term alone, within 3/4 units
    of 2^-53 of itself: a quarter for the term, and two coordinates, each within 2^-94 of the
    extent, where the term is 2^-13 of it (2^-54)."""
    exe = tmp_path / "fixcomp_check"
    subprocess.run(["g++", "-std=c++20", "-O2", "-ffp-contract=off",
                    f"-I{ROOT}/ode_prototyping_gb300/csrc",
                    os.path.join(ROOT, "tests", "cpp", "fixcomp_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    out = r.stdout.split()
    assert r.returncode == 0 and out[4] == "ok", (r.returncode, out)
    assert float(out[0]) <= 0.75 and int(out[1]) > 100000 and int(out[2]) > 10000, out
    # two words: 0.8 2^32 of a weight is 6.4 units of 2^-53 of 2^82 weights, the term half a unit
    assert float(out[3]) <= 8.75, out
