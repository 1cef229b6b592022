"""The compensated sums of the mixed form keep every product: rows whose large entries
cancel or outweigh 2^-24 of them (tests/cpp/mixed_sums_harness.cu, on the library's own
device code).

Each quad of a row adds 1 + 2^-25 + 2^-25 - 1 to an energy.  Compensated entry by entry every
term below is a multiple of 2^-25 under 2^-25 2^24, so the sum 2^-24 quads is exact; an
uncompensated addition within a quad gives 0.

A norm of quads (2^-13, 2^-13, 2^-13, 1) is sqrt(quads (1 + 3 2^-26)); its float-float sums are
exact to 2^-46 of it and the corrected square root to the square of FP32's half unit, 2^-48:
2^-44 of the norm.  Without compensation within a quad it errs by 2^-25.4."""
import math
import os
import subprocess

import pytest

from flare_pp_gb300 import build

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def harness(gpu_lib, tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("sums") / "harness")
    src = os.path.join(ROOT, "tests", "cpp", "mixed_sums_harness.cu")
    r = subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "-diag-suppress", "177",
                        "-I", build.CSRC, src, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


def run(harness, quads):
    r = subprocess.run([harness, str(quads)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    return {line.split()[0]: float(line.split()[1]) for line in r.stdout.splitlines()}


@pytest.mark.parametrize("quads", [1, 5, 32, 129, 400])
def test_energy(harness, quads):
    assert run(harness, quads)["energy"] == quads * 2.0 ** -24


@pytest.mark.parametrize("quads", [1, 5, 32, 129, 400])
def test_norm(harness, quads):
    want = math.sqrt(quads * (1 + 3 * 2.0 ** -26))
    assert abs(run(harness, quads)["norm"] - want) <= 2.0 ** -44 * want
