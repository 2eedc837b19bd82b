"""The Ritz stage's rotation (ql_rotation, ql.cuh) is rounded about as a norm and two
divisions are. Bounds, u = 2^-53: the sum of squares is off by at most 2 u, its root by
half of that and by the rounding of the corrected value: 2 u. A quotient by that and
its own rounding: 3 u. What the corrections leave out is of order u^2: 1%."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
HEADER = os.path.join(os.path.dirname(HERE), "ftlm_extended_hubbard_development_b200", "csrc", "ql.cuh")


def test_rotation_is_rounded_about_once(tmp_path):
    exe = str(tmp_path / "ql_rotation")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", '-DQL_HEADER="%s"' % HEADER,
                    os.path.join(HERE, "native", "ql_rotation.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout.split()
    assert float(out[0]) <= 2.0 * 1.01
    assert float(out[1]) <= 3.0 * 1.01
    assert int(out[2]) == 0
