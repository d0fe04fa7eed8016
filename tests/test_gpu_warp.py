"""The warp search kernel (variant 12, the default) on the GPU: the reference's lengths for every kind
and format at the smallest and at odd batch sizes, donations that search every node exactly once, and
positions whose search is wide (the superflip) in both table kinds."""

from __future__ import annotations

import pytest

from conftest import resident_handle
from cuda_cube_solver import native, workloads
from cuda_cube_solver.cubie import MOVES_HTM, CubieState, apply_moves
from cuda_cube_solver.device import state_words
from cuda_cube_solver.solver import parse_moves, verify_solutions

pytestmark = pytest.mark.gpu


def _words(cubes):
    return state_words([apply_moves(CubieState(), [MOVES_HTM[m] for m in parse_moves(c["scramble"])]) for c in cubes])


@pytest.mark.parametrize("kind,fmt", [("304", "block"), ("s4", "b3"), ("a4t", "block"), ("d4t", "b3")])
@pytest.mark.parametrize("first,count", [(0, 1), (1, 2), (3, 33)])
def test_lengths_of_every_kind(lengths_golden, kind, fmt, first, count):
    h = resident_handle(kind, fmt)
    cubes = lengths_golden["random1000"][first:first + count]
    words = _words(cubes)
    res = h.solve(words, native.solve_opts(timeout_s=300, variant=12))
    assert [r.length for r in res] == [c["length"] for c in cubes]
    assert verify_solutions(words, [list(r.moves[: r.length]) for r in res])
    assert h.last_solve_stats()[1] == sum(r.probes for r in res)


def test_donations_keep_lengths_and_iteration_nodes(lengths_golden):
    h = resident_handle("d4")
    cubes = lengths_golden["distance20"][:4] + [lengths_golden["hard19"]] + lengths_golden["random1000"][:26]
    words = _words(cubes)
    base = dict(timeout_s=300, variant=12, deeper_at=(1e18, 1e18))
    off = h.solve(words, native.solve_opts(steal=-1, **base))
    assert h.last_solve_donations() == 0
    for depth in (3, 1):
        on = h.solve(words, native.solve_opts(steal_depth=depth, steal_min_nodes=-1, steal_period=1, **base))
        assert h.last_solve_donations() > 0
        assert [r.length for r in on] == [r.length for r in off] == [c["length"] for c in cubes]
        for a, b in zip(on, off):
            assert list(a.iter_nodes[: a.length]) == list(b.iter_nodes[: b.length])


@pytest.mark.parametrize("kind", ["d4", "d4t"])
def test_superflip(kind):
    h = resident_handle(kind)
    words = state_words([workloads.superflip()])
    for base_plen in (1, 4):  # (1: items of 18 to 3,240 per iteration, split by donations)
        res = h.solve(words, native.solve_opts(timeout_s=300, base_plen=base_plen))
        assert res[0].length == 20 and verify_solutions(words, [list(res[0].moves[:20])])


def test_spilled_nodes_are_donated():
    """In items of fewer moves a wide search keeps its large subtrees in spill lists.  Were they not donated, the
    superflip's iterations would end on a few warps: 3.8 s on d4t with base_plen 3 against 2.5 s with 4, and
    2.7 s with them."""

    h = resident_handle("d4t")
    words, ms = state_words([workloads.superflip()]), {}
    for base_plen in (4, 3):
        res = h.solve(words, native.solve_opts(timeout_s=300, base_plen=base_plen))
        assert res[0].length == 20
        ms[base_plen] = h.last_solve_stats()[0]
    assert ms[3] < 1.3 * ms[4]
