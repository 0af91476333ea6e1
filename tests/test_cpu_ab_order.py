"""Host side of the alpha-beta schedule (csrc/ab_order.h), compiled for the CPU."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("ab_order") / "ab_order")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-pthread", "-fsanitize=undefined,float-divide-by-zero,float-cast-overflow",
                    "-fno-sanitize-recover=all", "-I" + os.path.join(ROOT, "sbd-ykt_b200", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "cpp", "ab_order.cc")], check=True)
    return out


@pytest.mark.parametrize("what", ["jobs", "order"])
def test_schedule(program, what):
    """jobs: an exception on a worker thread reaches the caller, with every
    thread joined (a host allocation that fails must not end the program).
    order: batches without lanes or singles, partial warps and crowded strings."""
    r = subprocess.run([program, what], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
