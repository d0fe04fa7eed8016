"""What the solver is timed on: the calls a program makes, through the package's public entry points.

A program opens a solver once, on a table that stays in device memory, and then brings it cubes:
one per call (the reference's drop-in shape), in batches, through the server, or through the call
that allocates nothing; and it builds tables.  The cases are those calls over the table kinds and
formats and from the smallest cubes (scrambles of 8 to 12 moves, solved in well under a
millisecond of search) to batches with positions of 19 moves and the superflip.

A solve's outputs are the optimal lengths and the positions that the returned moves reach.  The
moves themselves are not outputs: most cubes have several optimal solutions, and which of them is
found depends on the order in which the lanes finish.  All outputs are whole numbers.
"""

from __future__ import annotations

import sys
from pathlib import Path

import numpy as np

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "cuda-cube-solver_b200"))

from cuda_cube_solver import native, serving, table, workloads  # noqa: E402
from cuda_cube_solver.cubie import MOVES_HTM  # noqa: E402
from cuda_cube_solver.device import state_words  # noqa: E402
from cuda_cube_solver.solver import GpuSolver  # noqa: E402

# Table probes of one uniform random cube, by table (measured over 512 cubes of workloads seed 2);
# a probe needs one 32-byte sector of the table.
PROBES = {"304": 651e6, "s4-b3": 295e6, "a4t": 153e6, "d4t-b3": 101e6, "d4t": 92e6, "d4": 107e6}
SECTOR = 32
HARD_PROBES = 400e6  # a position of 19 moves on d4t
SUPERFLIP_PROBES = 13.5e9  # on d4
SCRAMBLE_PROBES = 2e3  # 8 to 12 moves
# Entries of the kinds that the build cases build, and entries per sector of each format.
ENTRIES = {"304": 5_505_192_000, "s4": 10_066_636_800}
PER_SECTOR = {"block": 124, "b3": 155}


def listed() -> list[dict]:
    return [
        # short scrambles, one per call: a trainer or a timer app checking what it was given
        dict(name="scrambles one by one", path="single", table="d4t", cubes="scramble", n=24),
        # the reference's own use: uniform cubes, one per call
        dict(name="cubes one by one", path="single", table="d4t", cubes="uniform", n=12),
        # a small batch: fewer cubes than fill the GPU
        dict(name="batch of 16", path="batch", table="d4t", cubes="uniform", n=16),
        # the reference's default chunk
        dict(name="batch of 100", path="batch", table="d4t", cubes="uniform", n=100),
        # the batched workload's mix: 5% of the cubes are positions of 19 moves
        dict(name="batch of 256, hard", path="batch", table="d4t", cubes="mix", n=256),
        # less device memory: the base-3 table, and the smallest preset
        dict(name="batch of 48, base 3", path="batch", table="d4t-b3", cubes="uniform", n=48),
        dict(name="batch of 20, 304", path="batch", table="304", cubes="uniform", n=20),
        # two resident tables, the superflip among ordinary cubes
        dict(name="two tables, superflip", path="dual", table="d4t", cubes="superflip", n=24),
        # a caller that cannot allocate device memory
        dict(name="no allocation, 64", path="noalloc", table="d4t", cubes="uniform", n=64),
        # a burst of requests through the server
        dict(name="served burst of 64", path="serve", table="d4t", cubes="uniform", n=64),
        # building the tables (and reading them: their histogram, bounds of cubes)
        dict(name="build 304", path="build", table="304", cubes="", n=65536),
        dict(name="build s4, base 3", path="build", table="s4-b3", cubes="", n=50021),
    ]


def _spread(rng, lo: int, hi: int) -> int:
    """A whole number of lo..hi, spread over its logarithm."""

    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def draw(rng) -> dict:
    path = rng.choice(["single", "single", "batch", "batch", "batch", "dual", "noalloc", "serve", "build"])
    if path == "build":
        return dict(path=path, table=rng.choice(["304", "304-b3", "s4", "s4-b3"]), cubes="", n=_spread(rng, 1, 100_000))
    if path == "dual":
        return dict(path=path, table="d4t", cubes="superflip", n=_spread(rng, 2, 40))
    if path == "single":
        if rng.random() < 0.5:
            return dict(path=path, table=rng.choice(sorted(PROBES)), cubes="scramble", n=_spread(rng, 4, 64))
        name = rng.choice(["d4t", "d4", "a4t", "d4t-b3"])
        return dict(path=path, table=name, cubes="uniform", n=_spread(rng, 3, 16))
    name = rng.choice(["d4t", "d4t", "d4", "a4t", "d4t-b3", "s4-b3", "304"])
    if path == "batch" and rng.random() < 0.2:
        return dict(path=path, table=name, cubes="scramble", n=_spread(rng, 2, 400))
    most = int(22e9 / PROBES[name])
    cubes = "mix" if path == "batch" and name == "d4t" and rng.random() < 0.4 else "uniform"
    return dict(path=path, table=name, cubes=cubes, n=_spread(rng, 2, min(most, 192)))


# A program keeps its solver: one per table (and one with the second table beside it).
_SOLVERS: dict[tuple[str, str | None], GpuSolver] = {}


def _kind_format(name: str) -> tuple[str, str]:
    return (name[:-3], "b3") if name.endswith("-b3") else (name, "block")


def _solver(name: str, second: str | None = None) -> GpuSolver:
    key = (name, second)
    if key not in _SOLVERS:
        kind, fmt = _kind_format(name)
        _SOLVERS[key] = GpuSolver.build_resident(kind, fmt, second_kind=second)
    return _SOLVERS[key]


_HARD: list = []


def _hard_cubes() -> list:
    """The positions of at least 19 moves that the package lists."""

    if not _HARD:
        at = workloads.hard20()["indices"][:96]
        stream = workloads.uniform_cubes(at[-1] + 1, seed=20)
        _HARD.extend(stream[i] for i in at)
    return _HARD


def _cubes(case: dict, seed: int) -> list:
    n, rng = case["n"], np.random.default_rng(seed)
    if case["cubes"] == "scramble":
        return [workloads.scramble_state(s) for s in workloads.small_scrambles(n, seed=seed)]
    cubes = workloads.uniform_cubes(n, seed=seed)
    if case["cubes"] == "superflip":
        cubes[int(rng.integers(n))] = workloads.superflip()
    if case["cubes"] == "mix":
        hard = _hard_cubes()
        at = rng.choice(n, size=max(1, round(0.05 * n)), replace=False)
        for i, j in zip(at, rng.choice(len(hard), size=len(at), replace=False)):
            cubes[int(i)] = hard[int(j)]
    return cubes


def _random_words(n: int, seed: int) -> np.ndarray:
    """Packed uniform random positions (n, 5), made for the whole array at once."""

    rng = np.random.default_rng(seed)
    cp, ep = rng.random((n, 8)).argsort(axis=1), rng.random((n, 12)).argsort(axis=1)
    inv = [sum((p[:, i] > p[:, j]).astype(int) for i in range(p.shape[1]) for j in range(i + 1, p.shape[1])) for p in (cp, ep)]
    odd = (inv[0] + inv[1]) % 2 == 1
    ep[odd, 10], ep[odd, 11] = ep[odd, 11].copy(), ep[odd, 10].copy()
    co, eo = rng.integers(0, 3, (n, 8)), rng.integers(0, 2, (n, 12))
    co[:, 7] = -co[:, :7].sum(axis=1) % 3
    eo[:, 11] = eo[:, :11].sum(axis=1) % 2
    return np.concatenate([cp | co << 3, ep | eo << 4], axis=1).astype(np.uint8).view(np.uint32).reshape(n, 5)


def prepare(case: dict, seed: int) -> dict:
    if case["path"] == "build":
        return dict(case=case, words=_random_words(case["n"], seed))
    solver = _solver(case["table"], "d4" if case["path"] == "dual" else None)
    cubes = _cubes(case, seed)
    state = dict(case=case, solver=solver, cubes=cubes, words=state_words(cubes))
    if case["path"] == "serve":
        state["arrivals"] = serving.poisson_arrivals(len(cubes), 10_000.0, seed=seed)
    return state


_CP = np.array([m.cp for m in MOVES_HTM] + [range(8)])
_CO = np.array([m.co for m in MOVES_HTM] + [[0] * 8])
_EP = np.array([m.ep for m in MOVES_HTM] + [range(12)])
_EO = np.array([m.eo for m in MOVES_HTM] + [[0] * 12])


def _outcome(words: np.ndarray, moves: list[list[int]]) -> dict:
    """The lengths, and the position that each cube's moves reach (its 20 packed bytes)."""

    b = words.view(np.uint8).reshape(-1, 20).astype(np.int64)
    cp, co, ep, eo = b[:, :8] & 7, b[:, :8] >> 3, b[:, 8:] & 15, b[:, 8:] >> 4
    for j in range(max(map(len, moves))):
        m = np.array([s[j] if j < len(s) else 18 for s in moves])
        cp, co = np.take_along_axis(cp, _CP[m], 1), (np.take_along_axis(co, _CP[m], 1) + _CO[m]) % 3
        ep, eo = np.take_along_axis(ep, _EP[m], 1), (np.take_along_axis(eo, _EP[m], 1) + _EO[m]) % 2
    reached = np.concatenate([cp | co << 3, ep | eo << 4], axis=1).astype(np.uint8)
    return {"lengths": np.array([len(s) for s in moves]), "reached": reached}


def _build(case: dict, words: np.ndarray) -> dict:
    kind, fmt = _kind_format(case["table"])
    solver = GpuSolver.build_resident(kind, fmt)
    out = {"counts": np.array(solver.build_counts), "histogram": np.array(table.histogram(solver.handle)),
           "bounds": solver.handle.lower_bound(words)}
    solver.close()
    return out


def run(state: dict):
    case = state["case"]
    if case["path"] == "build":
        return _build(case, state["words"])
    solver, cubes, words = state["solver"], state["cubes"], state["words"]
    if case["path"] == "single":
        moves = [solver.solve([c])[0].moves for c in cubes]
    elif case["path"] == "noalloc":
        moves = [list(r.moves[: r.length]) for r in solver.handle.solve_noalloc(words, native.solve_opts())]
    elif case["path"] == "serve":
        server = serving.Server(solver.handle, slots=1024)
        moves = [r.moves for r in serving.replay(server, cubes, state["arrivals"])["results"]]
        server.close()
    else:
        moves = [s.moves for s in solver.solve(cubes)]
    return _outcome(words, moves)


def work(case: dict) -> dict:
    """Bytes: a sector of the table for each probe of the method's search; a build writes its table
    once and reads it once (the histogram)."""

    n = case["n"]
    if case["path"] == "build":
        kind, fmt = _kind_format(case["table"])
        return {"bytes": 2 * SECTOR * -(-ENTRIES[kind] // PER_SECTOR[fmt]) + (20 + SECTOR + 4) * n, "flops": 0}
    probes = n * (SCRAMBLE_PROBES if case["cubes"] == "scramble" else PROBES[case["table"]])
    if case["cubes"] == "mix":
        probes += max(1, round(0.05 * n)) * (HARD_PROBES - PROBES[case["table"]])
    if case["cubes"] == "superflip":
        probes += SUPERFLIP_PROBES - PROBES["d4t"]
    return {"bytes": probes * SECTOR, "flops": 0}


def exact(case: dict, seed: int):
    """No output is a rounded number: lengths, positions, counts and bounds are whole and compared
    as they are."""

    return None
