"""The warp search kernel on the host (tests/emul/warp_emul.cpp): its probe arithmetic against the CPU
oracle for every kind, and whole searches of one emulated warp on an all-zero table, at full size and
with so few nodes and stash entries that the spill list carries most of the search."""

from __future__ import annotations

import ctypes
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from cuda_cube_solver import workloads
from cuda_cube_solver.cubie import MOVES_HTM, CubieState, apply_moves
from cuda_cube_solver.device import state_words
from cuda_cube_solver.prefixes import canonical_prefixes

KINDS = ["304", "s4", "d4f", "a4t", "d4t", "d4", "a4"]


@pytest.fixture(scope="module")
def libs():
    subprocess.run(["make", "-C", str(ROOT / "tests" / "emul"), "warp"], check=True, capture_output=True)
    return {v: ctypes.CDLL(str(ROOT / "_build" / "emul" / f"libccs_warp_{v}.so")) for v in ("full", "small", "tiny")}


@pytest.mark.parametrize("name", KINDS)
def test_probe_arithmetic_matches_oracle(libs, oracle, name):
    oracle.set_kind(name)
    words = oracle.unrank(np.random.default_rng(17).integers(0, oracle.n_entries(), 500, dtype=np.uint64))
    out = np.zeros(len(words), np.uint64)
    for m, left in [(-1, 0)] + [(m, left) for m in range(18) for left in (0, 1)]:
        assert libs["full"].emul_warp_index(name.encode(), ctypes.c_void_p(words.ctypes.data), len(words), m, left,
                                            ctypes.c_void_p(out.ctypes.data)) == 0
        assert np.array_equal(out, oracle.index(words, -2 - m if left else m)), (m, left)


def test_block_decode_of_every_entry(libs):
    sectors = np.random.default_rng(3).integers(0, 1 << 32, (124, 8), dtype=np.uint64).astype(np.uint32)
    entry, out = np.arange(124, dtype=np.uint32), np.zeros(124, np.uint32)
    libs["full"].emul_warp_decode(ctypes.c_void_p(sectors.ctypes.data), ctypes.c_void_p(entry.ctypes.data), 124,
                                  ctypes.c_void_p(out.ctypes.data))
    b = np.unpackbits(sectors.view(np.uint8), axis=1, bitorder="little")
    want = [int(sectors[j, 0] & 0xFF) + int(b[j, 8 + 2 * j]) + 2 * int(b[j, 9 + 2 * j]) for j in range(124)]
    assert out.tolist() == want


def test_base3_decode_of_every_byte_and_entry(libs):
    """Every value of a byte at every one of the 155 entries, against digits by division."""

    byte, entry = (a.ravel() for a in np.meshgrid(np.arange(256), np.arange(155), indexing="ij"))
    sectors = np.random.default_rng(4).integers(0, 256, (len(entry), 32), dtype=np.uint8)
    sectors[np.arange(len(entry)), 1 + entry // 5] = byte
    words, at, out = sectors.view(np.uint32).copy(), entry.astype(np.uint32), np.zeros(len(entry), np.uint32)
    libs["full"].emul_warp_decode_b3(*(ctypes.c_void_p(a.ctypes.data) for a in (words, at)), len(at), ctypes.c_void_p(out.ctypes.data))
    head = sectors[:, 0].astype(np.int64)
    digit = byte // 3 ** (entry % 5) % 3
    assert np.array_equal(out, (head & 63) + np.where(digit == 0, 0, (head >> 6) + digit))


@pytest.mark.parametrize("size", ["full", "small", "tiny"])
@pytest.mark.parametrize("name,starving", [("304", 0), ("s4", 1)])
def test_every_node_is_searched_once(libs, size, name, starving):
    """With all bounds zero nothing is pruned, so a completed iteration visits every canonical sequence
    up to its bound (a prefix's moves once per item): the counts tell a lost or repeated node.  The
    prefix lengths for bounds 1 to 4 are 1, 2, 3 and 4 moves, with donations 1, 1, 2 and 3."""

    scrambles = [s[:4] for s in workloads.small_scrambles(2, seed=5)]
    states = [workloads.scramble_state(s) for s in scrambles] + [CubieState()]
    words, n = state_words(states), len(states)
    lengths, moves = np.zeros(n, np.uint32), np.zeros((n, 24), np.uint8)
    nodes, donated = np.zeros((n, 24), np.uint64), ctypes.c_uint64()
    ptr = [ctypes.c_void_p(a.ctypes.data) for a in (words, lengths, moves, nodes)]
    assert libs[size].emul_warp_solve(name.encode(), ptr[0], n, starving, ptr[1], ptr[2], ptr[3], ctypes.byref(donated)) == 0
    count = [len(canonical_prefixes(L)) for L in range(5)]
    full = {1: count[1], 2: 2 * count[2], 3: 3 * count[3]}
    if starving:
        full = {1: count[1], 2: count[1] + count[2], 3: 2 * count[2] + count[3]}
    for s, length, mv, it in zip(states, lengths, moves, nodes):
        assert length <= 4 and apply_moves(s, [MOVES_HTM[m] for m in mv[:length]]) == CubieState()
        assert [int(it[b]) for b in range(1, length)] == [full[b] for b in range(1, length)]
    assert lengths[-1] == 0 and max(lengths) == 4
    assert not starving or donated.value > 0


def test_items_of_a_solved_cube_are_dropped_together(libs):
    """The iteration that finds a cube's solution hands out up to millions of items; the ones left are counted
    as done at once, not fetched one by one (43,254 of them here; a fetch is some 35 of the warp's steps)."""

    back = [0, 4, 8, 9, 13]  # (an early one of the items)
    state = apply_moves(CubieState(), [MOVES_HTM[3 * (m // 3) + 2 - m % 3] for m in reversed(back)])
    words, length, moves = state_words([state]), np.zeros(1, np.uint32), np.zeros(24, np.uint8)
    nodes, donated = np.zeros(24, np.uint64), ctypes.c_uint64()
    ptr = [ctypes.c_void_p(a.ctypes.data) for a in (words, length, moves, nodes)]
    assert libs["full"].emul_warp_solve(b"s4", ptr[0], 1, 0, ptr[1], ptr[2], ptr[3], ctypes.byref(donated)) == 0
    libs["full"].emul_warp_turns.restype = ctypes.c_uint64
    assert length[0] == 5 and libs["full"].emul_warp_turns() < 20 * len(canonical_prefixes(4))


SLOT_SOLVED, SLOT_ERROR, ERR_STACK, ERR_STUCK = 2, 3, 4, 8


@pytest.mark.parametrize("back", [[17, 13, 8, 3], [17, 13, 8, 3, 0, 5, 16]])
def test_a_full_spill_list_fails_the_cube(libs, back):
    """With room for 32 spilled nodes an iteration of four moves drops subtrees: the cube ends there as an error,
    it is not searched on for a longer solution.  One found in that iteration all the same is optimal."""

    state = apply_moves(CubieState(), [MOVES_HTM[3 * (m // 3) + 2 - m % 3] for m in reversed(back)])
    lib = ctypes.CDLL(str(ROOT / "_build" / "emul" / "libccs_warp_over.so"))
    words, status, length, moves = state_words([state]), np.zeros(1, np.uint32), np.zeros(1, np.uint32), np.zeros(24, np.uint8)
    nodes, donated = np.zeros(24, np.uint64), ctypes.c_uint64()
    ptr = [ctypes.c_void_p(a.ctypes.data) for a in (words, status, length, moves, nodes)]
    assert lib.emul_warp_search(b"s4", ptr[0], 1, 2, *ptr[1:], ctypes.byref(donated)) == ERR_STACK
    if len(back) > 4 or status[0] != SLOT_SOLVED:
        assert status[0] == SLOT_ERROR
    else:
        assert length[0] == 4
    assert nodes[4] > 0 and nodes[5:].sum() == 0


def test_a_warp_that_gives_up_fails_the_cube(libs):
    """A warp that makes no progress drops its work and counts its units as done, so that the cube ends in an
    error (a served one would otherwise never end)."""

    lib = ctypes.CDLL(str(ROOT / "_build" / "emul" / "libccs_warp_stuck.so"))
    state = workloads.scramble_state(workloads.small_scrambles(1, seed=5)[0])
    words, status, length, moves = state_words([state]), np.zeros(1, np.uint32), np.zeros(1, np.uint32), np.zeros(24, np.uint8)
    nodes, donated = np.zeros(24, np.uint64), ctypes.c_uint64()
    ptr = [ctypes.c_void_p(a.ctypes.data) for a in (words, status, length, moves, nodes)]
    assert lib.emul_warp_search(b"s4", ptr[0], 1, 0, *ptr[1:], ctypes.byref(donated)) == ERR_STUCK
    assert status[0] == SLOT_ERROR


def test_a_nearly_full_spill_list_narrows_the_search(libs):
    """With room for 96 spilled nodes and one child at a time from 10 on, a search that would hold more than 96 (the
    list overflows without that rule) keeps within its list and still visits every node once."""

    back = [17, 13, 8, 3]
    state = apply_moves(CubieState(), [MOVES_HTM[3 * (m // 3) + 2 - m % 3] for m in reversed(back)])
    lib = ctypes.CDLL(str(ROOT / "_build" / "emul" / "libccs_warp_narrow.so"))
    words, status, length, moves = state_words([state]), np.zeros(1, np.uint32), np.zeros(1, np.uint32), np.zeros(24, np.uint8)
    nodes, donated = np.zeros(24, np.uint64), ctypes.c_uint64()
    ptr = [ctypes.c_void_p(a.ctypes.data) for a in (words, status, length, moves, nodes)]
    assert lib.emul_warp_search(b"s4", ptr[0], 1, 2, *ptr[1:], ctypes.byref(donated)) == 0
    assert status[0] == SLOT_SOLVED and length[0] == 4
    count = np.cumsum([len(canonical_prefixes(L)) for L in range(1, 4)])  # (items of one move)
    assert nodes[1:4].tolist() == count.tolist()
