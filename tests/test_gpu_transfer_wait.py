"""Transfers share pinned slots and helper threads only while they copy: a read
that waits for its own reconstruction's iterations keeps nobody else waiting."""
import threading
import time

import numpy as np
import pytest

import pynadia
from pynadia import FP32, FP64

pytestmark = pytest.mark.gpu


def reconstruction(n, prec, seed):
    g = np.random.default_rng(seed)
    s = pynadia.Solver("planar", n, n, precision=prec)
    sup = np.zeros((n, n))
    sup[n // 4:n // 2, n // 4:n // 2] = 1
    s.set_support(sup)
    s.set_intensity(g.random((n, n)) + 1)
    s.set_exit_surface_wave(sup + 0j)
    s.set_algorithm("HIO")
    return s


@pytest.mark.parametrize("prec", [FP32, FP64])
def test_idle_upload_beside_queued_reads(prec):
    """Nine reads (with the helpers more threads than there are slots) behind
    iterations that take hundreds of milliseconds; an idle reconstruction's
    upload is done before the first of them."""
    readers = [reconstruction(1024, FP32, k) for k in range(9)]
    idle = reconstruction(1024, prec, 99)
    x = np.random.default_rng(100).random((1024, 1024)) + 0j
    idle.set_exit_surface_wave(x)
    for h in readers:
        h.iterate(10)
        h.get_error()
    queued = threading.Barrier(len(readers) + 1)
    ends, errors = [], []

    def read(h):
        try:
            h.iterate(8000)
            queued.wait()
            h.get_exit_surface_wave()
            ends.append(time.perf_counter())
        except Exception as e:  # reported by the main thread
            errors.append(e)

    ts = [threading.Thread(target=read, args=(h,)) for h in readers]
    for t in ts:
        t.start()
    queued.wait()
    time.sleep(0.02)  # the reads are waiting
    idle.set_exit_surface_wave(x)
    uploaded = time.perf_counter()
    for t in ts:
        t.join()
    assert not errors, errors
    assert uploaded < min(ends), (uploaded - min(ends), max(ends) - min(ends))
