"""tpcf_loop_units against the loops it stands for, counted one by one: every
kind and loop nest, catalogs of unlike sizes, and ranges whose end lies before
their begin (the entry point takes them: their loops do not run)."""
import itertools

import numpy as np
import pytest

import tpcf

pytestmark = pytest.mark.gpu


def _loops(kind, loop, n):
    if kind == tpcf.PAIR:
        if loop != tpcf.LOOP_SAME:
            return n[0] * n[1]
        return sum(max(n[1] - i, 0) for i in range(n[0]))
    if kind == tpcf.THREE_SIDE or loop == tpcf.LOOP_ALL:
        return n[0] * n[1] * n[2]
    return sum((min(n[0], j + 1) if loop == tpcf.LOOP_SAME else n[0]) * max(n[2] - j, 0) for j in range(n[1]))


def test_closed_forms():
    axes = [(8, 2.0, 10.0), (8, 1.0, 3.0), (16, 0.0, 1.0)]
    with tpcf.Engine(0) as eng:
        h = eng.catalog(np.zeros((40, 3), np.float32))
        for n in itertools.product((-3, 0, 1, 2, 7, 20), repeat=3):
            ranges = [(10, 10 + x) for x in n]
            for kind, loop in itertools.product((tpcf.PAIR, tpcf.TRIANGLE, tpcf.TRIANGLE_JBJ, tpcf.THREE_SIDE),
                                                (tpcf.LOOP_ALL, tpcf.LOOP_SAME, tpcf.LOOP_ONE)):
                spec = tpcf.make_spec(kind, loop, axes)
                assert eng.loop_units(spec, eng.job([h] * 3, ranges)) == _loops(kind, loop, n) % 2**64, (kind, loop, n)


def test_sizes_of_billions():
    """Sums modulo 2^64 (the ranges are only measured, not looked up)."""
    with tpcf.Engine(0) as eng:
        h = eng.catalog(np.zeros((40, 3), np.float32))
        for n in itertools.product((1, 999_999_937, 2**30 - 1, 2**30), repeat=3):
            job = eng.job([h] * 3, [(0, x) for x in n])
            m = min(n[1], n[2])
            tail = m * n[2] - m * (m - 1) // 2
            p = min(m, n[0])
            lin, sq = p * (p - 1) // 2, (p - 1) * p * (2 * p - 1) // 6
            same = p * n[2] + n[2] * lin - lin - sq + n[0] * (tail - (p * n[2] - lin))
            axes = [(8, 2.0, 10.0), (8, 1.0, 3.0), (16, 0.0, 1.0)]
            assert eng.loop_units(tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_ONE, axes), job) == n[0] * tail % 2**64
            assert eng.loop_units(tpcf.make_spec(tpcf.TRIANGLE, tpcf.LOOP_SAME, axes), job) == same % 2**64
            k = min(n[0], n[1])
            assert eng.loop_units(tpcf.make_spec(tpcf.PAIR, tpcf.LOOP_SAME, axes), job) == (k * n[1] - k * (k - 1) // 2) % 2**64
