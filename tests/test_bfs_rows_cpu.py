"""The table build's kernels on the host (tests/emul/rows_emul.cpp): where a dense pass looks for an
entry's neighbours, against the CPU oracle's unrank, move and index for every kind and move; and the
encoders on made-up distances, against a plain count of what the formats say."""

from __future__ import annotations

import ctypes
import subprocess

import numpy as np
import pytest

from conftest import ROOT

KINDS = ["304", "s4", "d4f", "a4t", "d4t", "d4", "a4"]


@pytest.fixture(scope="module")
def rows():
    subprocess.run(["make", "-C", str(ROOT / "tests" / "emul"), "rows"], check=True, capture_output=True)
    return ctypes.CDLL(str(ROOT / "_build" / "emul" / "libccs_rows.so"))


def _ptr(a):
    return ctypes.c_void_p(a.ctypes.data)


@pytest.mark.parametrize("name", KINDS)
def test_neighbours_match_oracle(rows, oracle, name):
    oracle.set_kind(name)
    n = oracle.n_entries()
    idx = np.concatenate([[0, n - 1], np.random.default_rng(23).integers(0, n, 600, dtype=np.uint64)]).astype(np.uint64)
    states, out = oracle.unrank(idx), np.zeros(len(idx), np.uint64)
    for m in range(18):
        assert rows.emul_rows_neighbours(name.encode(), _ptr(idx), len(idx), m, _ptr(out)) == 0
        assert np.array_equal(out, oracle.index(states, m)), m


def _block(d):
    out = np.zeros((-(-len(d) // 124), 32), np.uint8)
    for b in range(len(out)):
        v = d[124 * b: 124 * b + 124].astype(int)
        out[b, 0] = v.min()
        for j, o in enumerate(np.minimum(v - v.min(), 3)):
            out[b, 1 + j // 4] |= int(o) << (2 * (j % 4))
    return out


def _b3(d):
    m124 = np.repeat([int(d[i: i + 124].min()) for i in range(0, len(d), 124)], 124)[: len(d)]
    x = d.astype(int)
    x = np.where(x <= m124 + 5, x, m124 + 3 + (x - m124 - 3) % 3)
    out = np.zeros((-(-len(d) // 155), 32), np.uint8)
    for b in range(len(out)):
        v = x[155 * b: 155 * b + 155]
        m = v.min()
        coded = [np.where(v <= m + c, m, np.where(v == m + c + 1, m + c + 1, m + c + 2)) for c in range(4)]
        c = int(np.argmax([s.sum() for s in coded]))
        digit = np.where(v <= m + c, 0, np.where(v == m + c + 1, 1, 2))
        out[b, 0] = m | c << 6
        for j, g in enumerate(digit):
            out[b, 1 + j // 5] += int(g) * 3 ** (j % 5)
    return out


@pytest.mark.parametrize("name", ["304", "s4", "a4t", "d4f", "d4t"])
@pytest.mark.parametrize("n,top", [(1, 14), (123, 14), (124, 9), (155, 14), (156, 3), (5000, 14), (4999, 28)])
def test_encoders(rows, name, n, top):
    rng = np.random.default_rng(n)
    d = np.minimum(top, np.repeat(rng.integers(0, top, -(-n // 200)), 200)[:n] + rng.integers(0, 9, n)).astype(np.uint8)
    blk, b3 = np.zeros((-(-n // 124), 32), np.uint8), np.zeros((-(-n // 155), 32), np.uint8)
    mod3 = np.zeros(-(-n // 16), np.uint32)
    assert rows.emul_rows_encode(name.encode(), _ptr(d), ctypes.c_uint64(n), int(top > 14), _ptr(blk), _ptr(b3), _ptr(mod3)) == 0
    assert np.array_equal(blk, _block(d))
    assert np.array_equal(b3, _b3(d))
    r = np.concatenate([d % 3, np.full(-n % 16, 3)]).reshape(-1, 16).astype(np.uint64)
    assert np.array_equal(mod3, (r << (2 * np.arange(16, dtype=np.uint64))).sum(axis=1).astype(np.uint32))


@pytest.mark.parametrize("name,columns,block_rows", [("304", 16, 70), ("s4", 8, 256), ("d4f", 12, 256), ("a4t", 16, 256), ("d4t", 24, 256)])
@pytest.mark.parametrize("d", [0, 7, 13])
def test_frontier_read_off_the_planes(rows, name, columns, block_rows, d):
    """The frontier of a pass that claimed more entries than its list holds: the bits of every entry of that
    distance, and the flags of the blocks that have one."""

    per_block = columns * block_rows
    dist = np.random.default_rng(d).integers(0, 16, 3 * per_block).astype(np.uint8)
    dist[per_block: 2 * per_block][dist[per_block: 2 * per_block] == d] = 15  # a block without any
    bits, flags = np.zeros(len(dist), np.uint8), np.zeros(3, np.uint8)
    assert rows.emul_rows_mark(name.encode(), _ptr(dist), ctypes.c_uint64(len(dist)), d, _ptr(bits), _ptr(flags)) == 0
    assert np.array_equal(bits, dist == d) and flags.tolist() == [1, 0, 1]
