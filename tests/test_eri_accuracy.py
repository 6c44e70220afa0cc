"""Rounding errors of the light classes' building blocks (csrc/cuda/eri_low.cuh),
compiled for the host, against 113-bit references."""
import os
import subprocess

import pytest

from conftest import ROOT

HOST = os.path.join(ROOT, "tests", "host")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("host") / "eri_accuracy")
    # multiplications and additions contract, as nvcc does by default
    subprocess.run(["g++", "-std=gnu++17", "-O2", "-mfma", "-ffp-contract=fast", "-w", "-I" + os.path.join(HOST, "cuda"),
                    "-I" + os.path.join(ROOT, "gtfock_b200", "csrc", "cuda"), os.path.join(HOST, "eri_accuracy.cpp"),
                    "-o", exe, "-lquadmath"], check=True)
    return exe


def _run(*cmd):
    out = subprocess.run(cmd, check=True, capture_output=True, text=True).stdout
    return [[float(x) for x in line.split()] for line in out.splitlines()]


def test_boys_functions(program):
    """F_0 .. F_4 at interval edges, midpoints, random arguments and both sides
    of the large-T form: 3 units in the last place below it; above, 1/T and
    the product of m factors add one unit per m."""
    rows = _run(program, "boys")
    assert len(rows) == 10
    for m, bits, below, above in rows:
        assert below < 6.0, (m, bits)
        assert above < 4.0 + 2.0 * m, (m, bits)
