"""Device functions of the span kernels by themselves (tests/native/span_check.cu), for what a whole search
shows only after a fault."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NATIVE = os.path.join(ROOT, "tests", "native")
BIN = os.path.join(NATIVE, "_build", "span_check")


def _run(case):
    if not os.path.exists(BIN):
        subprocess.run(["make", "-s", "-C", NATIVE, BIN], check=True)
    r = subprocess.run([BIN, case], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return [int(v) for v in r.stdout.split()]


def test_every_part_reports_a_bad_address(cuda, lib):
    """The self-checking build's status bit of a part that is not the one to complete its task."""
    first, after, last, status = _run("bounds")
    assert (first, last) == (0, 1)
    assert after == status == 0x100
