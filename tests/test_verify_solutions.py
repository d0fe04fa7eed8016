"""The host check of returned solutions: both of its forms against the moves applied to cubie states."""

from __future__ import annotations

import numpy as np
import pytest

from cuda_cube_solver import workloads
from cuda_cube_solver.cubie import MOVES_HTM, CubieState, apply_moves
from cuda_cube_solver.device import state_words
from cuda_cube_solver.solver import verify_solutions


@pytest.mark.parametrize("n", [1, 12, 13, 60])
def test_right_and_wrong_solutions(n):
    rng = np.random.default_rng(n)
    moves = [[int(m) for m in rng.integers(0, 18, rng.integers(0, 21))] for _ in range(n)]
    states = [apply_moves(CubieState(), [MOVES_HTM[m] for m in s]) for s in moves]
    back = [[3 * (m // 3) + 2 - m % 3 for m in reversed(s)] for s in moves]
    words = state_words(states)
    assert verify_solutions(words, back)
    assert verify_solutions(words, [s + [-1] for s in back])  # a negative entry is no move
    at = int(rng.integers(n))
    for wrong in (back[at] + [int(rng.integers(18))], (back[at] + [3, 3, 3])):
        assert not verify_solutions(words, back[:at] + [wrong] + back[at + 1:])
    # every orientation counts: uniform cubes are solved by nothing
    assert not verify_solutions(state_words(workloads.uniform_cubes(n, seed=n)), [[] for _ in range(n)])
    with pytest.raises(IndexError):
        verify_solutions(words, back[:at] + [back[at] + [18]] + back[at + 1:])


@pytest.mark.parametrize("n", [1, 12, 13, 60])
def test_moves_for_another_number_of_cubes_are_refused(n):
    words = state_words([apply_moves(CubieState(), [MOVES_HTM[0]])] * n)
    assert verify_solutions(words, [[2]] * n)
    for other in {1, n - 1, n + 1} - {n, 0}:
        with pytest.raises(IndexError):
            verify_solutions(words, [[2]] * other)
    # a wrong move is refused wherever it stands, and moves may be any kind of number
    with pytest.raises(IndexError):
        verify_solutions(words, [[0]] * (n - 1) + [[0, 18]])
    assert verify_solutions(words, [[2.0]] * n)
