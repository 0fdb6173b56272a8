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


def test_a_task_with_a_lost_part_has_no_costs(cuda, lib):
    """A part that a CTA which gave up did not run: the task is retired with the timeout status, by whichever
    comes last, and its totals, never written, form no cost."""
    out = _run("lost")
    for joined, done, status, untouched in (out[:4], out[4:]):
        assert (joined, done, untouched) == (0, 1, 1)
        assert status == 7  # CGS_ERROR_DEVICE_TIMEOUT


def test_quotients_are_correctly_rounded(cuda, lib):
    """exact_quot2 over 3.9e9 quotients: ends of the binade, few and many bits, mixed mantissas, exponents over
    the range that quot_range admits."""
    tried, wrong = _run("quotients")
    assert tried > 3_000_000_000
    assert wrong == 0
