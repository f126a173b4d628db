"""The host helper threads alone, without a GPU: threads that make and drop the
last reconstruction at the same time neither hang nor lose work."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "nadia-coecxs_b200", "csrc")


def stress(tmp_path, linger_ms):
    exe = str(tmp_path / ("stress%d" % linger_ms))
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-DNADIA_HELPER_LINGER_MS=%d" % linger_ms,
                    "-I", CSRC, os.path.join(ROOT, "tests", "helpers_stress.cpp"),
                    os.path.join(CSRC, "helpers.cpp"), "-o", exe], check=True)
    return exe


# helpers that end as soon as they are unused, within the sleeps of the rounds,
# and never while the test runs
@pytest.mark.parametrize("linger_ms", [0, 1, 60000])
def test_last_users_at_once(tmp_path, linger_ms):
    exe = stress(tmp_path, linger_ms)
    for workers in ("1", "2", "1", "2"):
        # a hang ends in subprocess.TimeoutExpired
        r = subprocess.run([exe, "2", workers], stdout=subprocess.PIPE, text=True, timeout=60)
        assert r.returncode == 0, r.stdout
        rounds = int(r.stdout.split()[0])
        assert rounds > 100, r.stdout


def test_forked_child_ends(tmp_path):
    """A child forked while helpers sleep has none of them and still ends."""
    r = subprocess.run([stress(tmp_path, 60000), "0.2", "1", "fork"], stdout=subprocess.PIPE, text=True,
                       timeout=60)
    assert r.returncode == 0, r.stdout


def test_given_back_once_unused(tmp_path):
    exe = str(tmp_path / "give_back")
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-DNADIA_HELPER_LINGER_MS=200", "-I", CSRC,
                    os.path.join(ROOT, "tests", "helpers_give_back.cpp"),
                    os.path.join(CSRC, "helpers.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], stdout=subprocess.PIPE, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


# helpers wanted by a call, calls at once, and the most helpers that may run
@pytest.mark.parametrize("extra,calls,most", [(1, 1, 1), (2, 1, 2), (7, 1, 7), (7, 4, 16)])
def test_started_as_wanted(tmp_path, extra, calls, most):
    exe = str(tmp_path / "count")
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", CSRC,
                    os.path.join(ROOT, "tests", "helpers_count.cpp"),
                    os.path.join(CSRC, "helpers.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe, str(extra), str(calls)], stdout=subprocess.PIPE, text=True, timeout=60)
    assert r.returncode == 0
    assert min(1, os.cpu_count() // 2) <= int(r.stdout) <= min(most, max(1, os.cpu_count() // 2)), r.stdout
