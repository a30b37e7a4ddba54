"""The DP launch's item list (CPU only)."""
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def flow_check(tmp_path_factory):
    out = tmp_path_factory.mktemp("flow")
    subprocess.run(["gcc", "-O2", "-c", os.path.join(REPO, "oracle", "xted_oracle.c"), "-o", str(out / "xo.o")], check=True)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I/usr/local/cuda/include", os.path.join(REPO, "tests", "cpp", "flow_check.cpp"),
                    str(out / "xo.o"), "-o", str(out / "flow_check"), "-lpthread"], check=True)
    return str(out / "flow_check")


@pytest.mark.parametrize("rounds,nodes,seed", [("90", "60", "1"), ("30", "420", "2"), ("6", "700", "6")])
def test_items_read_what_was_written_before(flow_check, rounds, nodes, seed):
    """Items run in list order, whole and in parts that share the hand-off
    buffer (tests/cpp/flow_check.cpp): every word read was written before,
    every word is written once, distances are the oracle's."""
    r = subprocess.run([flow_check, rounds, nodes, seed], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("ok")
