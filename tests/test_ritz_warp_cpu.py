"""The Ritz stage's warp form of the implicit QL: its result may not depend on how the
lanes of the warp are scheduled (the engine's diagonaliser of each random vector's
tridiagonal, main.cpp:913-994)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ftlm_extended_hubbard_development_b200", "csrc")


def test_lanes_need_not_run_in_step(tmp_path):
    exe = str(tmp_path / "ql_warp")
    header = os.path.join(CSRC, "ql.cuh")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", f'-DQL_HEADER="{header}"',
                    os.path.join(HERE, "native", "ql_warp.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe, "25"], check=True, capture_output=True, text=True, timeout=300)
    assert int(out.stdout) == 0, f"{out.stdout.strip()} of 25 matrices depend on the lanes' order"
