"""Rounding errors of the light classes' integrals (csrc/cuda/eri_low.cuh),
compiled for the host, against 113-bit references: no larger than those of
Rys quadrature in the same precision, FP64 and FP32."""
import os
import subprocess

import pytest

from conftest import ROOT

HOST = os.path.join(ROOT, "tests", "host")
CLASSES = ["ssss", "psss", "psps", "ppss", "dsss", "dsps", "ppps", "dpss", "dpps", "dspp", "dsds", "ddss"]


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


@pytest.mark.parametrize("c", range(len(CLASSES)), ids=CLASSES)
def test_light_classes_are_no_less_accurate_than_rys(program, c):
    """Geometric mean over 150 random contracted quartets.  The two forms see
    the same quartets; a spread of a factor of 2.5 per quartet leaves 7% on
    the mean, so 1.15 means equal.  FP32: the errors of the Rys form times the
    ratio of the two roundings (2^29)."""
    e64_rys, e64, e32 = _run(program, "eri", str(c), "150")[0][4:]
    assert e64 < 1.15 * e64_rys
    assert e32 < 1.15 * 2.0 ** 29 * e64_rys


def test_boys_functions(program):
    """F_0 .. F_4 at interval edges, midpoints, random arguments and both sides
    of the large-T form: 3 units in the last place below it; above, 1/T and
    the product of m factors add one unit per m."""
    rows = _run(program, "boys")
    assert len(rows) == 10
    for m, bits, below, above in rows:
        assert below < 6.0, (m, bits)
        assert above < 4.0 + 2.0 * m, (m, bits)
