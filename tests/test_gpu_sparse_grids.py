"""Pair lists on grids with more cells than particles (and about as many):
the same neighbours and sums as the FP64 cell sweep, and no cost that grows
with the empty cells beyond that of the cell build itself."""
import time

import numpy as np
import pytest

import ggem_gb300 as G

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from ggem_gb300 import build as B
    B.build()


@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("n", [1, 2, 124, 125, 126, 900])  # 125 cells
def test_lists_around_one_particle_per_cell(n, symmetric):
    L = 36.0
    rng = np.random.default_rng(n)
    xyz = rng.uniform(0.0, L, (n, 3))
    xyz[: n // 2] = xyz[: n // 2] * 0.2  # half of them crowded into a few cells
    f = rng.standard_normal((n, 3))
    with G.Context(box_hi=(L,) * 3, precision=G.FP64) as c64, \
            G.Context(box_hi=(L,) * 3, precision=G.FP32) as c32:
        c64.set_fp64_pair_list(False)
        c32.set_pair_tensors(False)
        if symmetric:
            c32.set_symmetric_pairs(True)
        for c in (c64, c32):
            c.set_particles(xyz)
            c.build_cells()
        o64, i64 = c64.neighbors()
        o32, i32 = c32.neighbors()
        assert np.array_equal(o64, o32) and np.array_equal(i64, i32)
        want = c64.local_matvec(f)
        got = c32.local_matvec(f)
        # FP32 tensors of up to n pairs: 1e-6 as elsewhere for this path
        assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)


def test_empty_cells_cost_no_more_than_the_sweep():
    n, L = 2000, 1500.0  # 9.8e6 cells
    rng = np.random.default_rng(1)
    xyz, f = rng.uniform(0.0, L, (n, 3)), rng.standard_normal((n, 3))
    best = {}
    for own in (True, False):
        with G.Context(box_hi=(L,) * 3, precision=G.FP64) as c:
            if not own:
                c.set_fp64_pair_list(False)
            for _ in range(12):
                t0 = time.perf_counter()
                c.set_particles(xyz)
                c.build_cells()
                c.local_matvec(f)
                t = time.perf_counter() - t0
                best[own] = min(best.get(own, t), t)
    # (25 times as long when every empty cell took a block)
    assert best[True] <= 2.0 * best[False]
