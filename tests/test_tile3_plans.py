"""CPU check of PolyCDI's three-pass tiles (nadia-coecxs_b200/csrc/fused32_poly3.cuh):
the index algebra of every registered Tile3 -- which thread takes which
butterfly, twiddle exponents, exchange addresses, output positions -- replayed
for both maps and directions against numpy's DFT.  Every exchange writes each
word of the tile once, no twiddle index passes the table, and the values
leaving one direction sit where the other starts."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "nadia-coecxs_b200", "csrc")
TILES = [tuple(map(int, m)) for m in
         re.findall(r"Tile3<(\d+), (\d+), (\d+), (\d+), \d+>",
                    open(os.path.join(CSRC, "fused32_poly.cu")).read())]
L = 4


def deal(rows, edge, b):
    if rows and edge:
        return b // 4 % 4, b // 16 * 4 + b % 4
    return b % 4, b // 4


def test_there_are_tiles():
    assert TILES


@pytest.mark.parametrize("tile", TILES)
@pytest.mark.parametrize("rows", [True, False])
@pytest.mark.parametrize("fwd", [True, False])
def test_plan(tile, rows, fwd):
    n, ra, rb, rc = tile
    radices = (rc, rb, ra) if fwd else (ra, rb, rc)
    sign = -1 if fwd else 1
    g = np.random.default_rng(1)
    x = g.standard_normal((L, n)) + 1j * g.standard_normal((L, n))
    out, sm, span = np.zeros((L, n), complex), None, 1
    for p, r in enumerate(radices):
        nr = n // r
        new, seen = np.full(n * L, np.nan, complex), set()
        dft = np.exp(sign * 2j * np.pi * np.outer(np.arange(r), np.arange(r)) / r)
        for b in range(nr * L):
            s, j = deal(rows, p != 1, b)
            assert j < nr and (s, j) not in seen
            seen.add((s, j))
            at = j + np.arange(r) * nr
            v = x[s, at] if p == 0 else sm[at * L + s]
            t1 = j % span * (n // (span * r))
            assert t1 * (r - 1) < n
            y = dft @ (v * np.exp(sign * 2j * np.pi * t1 * np.arange(r) / n))
            if p < 2:
                new[((j // span) * span * r + j % span + np.arange(r) * span) * L + s] = y
            else:
                out[s, at] = y
        if p < 2:
            assert not np.isnan(new).any()
            sm = new
        span *= r
    ref = np.fft.fft(x, axis=1) if fwd else np.fft.ifft(x, axis=1) * n
    assert np.abs(out - ref).max() < 1e-13 * np.abs(ref).max()
