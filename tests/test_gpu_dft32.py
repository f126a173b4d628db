"""The packed forms of the short FP32 transforms are no further from 64 bits than
the scalar ones, in which the compiler contracts products into the sums after
them."""
import importlib.util
import math
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SAMPLES = 1 << 18


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    path = os.path.join(ROOT, "nadia-coecxs_b200", "build.py")
    spec = importlib.util.spec_from_file_location("nadia_build", path)
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    exe = str(tmp_path_factory.mktemp("dft32") / "dft32")
    subprocess.run([b.NVCC, *b.COMMON, os.path.join(ROOT, "tests", "dft32_error.cu"), "-o", exe],
                   check=True)
    out = subprocess.run([exe], stdout=subprocess.PIPE, text=True, check=True, timeout=120).stdout
    return [line.split() for line in out.splitlines()]


def test_packed_error_is_no_larger(rows):
    assert len(rows) == 20
    for radix, direction, packed, scalar in rows:
        packed, scalar = float(packed), float(scalar)
        # the same inputs to both; the spread of an error's root mean square over
        # 2 * radix * SAMPLES values, three times
        spread = 3 / math.sqrt(2 * 2 * int(radix) * SAMPLES)
        assert packed <= scalar * (1 + spread), (radix, direction, packed, scalar)
        # sums of two 24-bit fixed-point inputs are exact
        assert packed > 0 or radix == "2"
