"""The Lanczos recurrence where it ends before k steps: the bounds of the
steps that it has, at the cost of about those."""
import numpy as np
import pytest

import ggem_gb300 as G

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from ggem_gb300 import build as B
    B.build()


def _launches(ctx, k):
    a = ctx.launch_count()
    bounds = ctx.lanczos_bounds(k=k, seed=5)
    return ctx.launch_count() - a, bounds


@pytest.mark.parametrize("precision", [G.FP64, G.FP32])
@pytest.mark.parametrize("n", [1, 3, 343])
def test_ends_with_one_eigenvalue(n, precision):
    """no pair within the cut-off: M = c I, one step, for every k"""
    side = round(n ** (1 / 3)) if n == 343 else n
    L = 30.0 * max(side, 1)
    g = (np.arange(side) + 0.5) * 30.0
    xyz = np.stack(np.meshgrid(g, g, g), -1).reshape(-1, 3)[:n]
    with G.Context(box_hi=(max(L, 30.0),) * 3, precision=precision) as ctx:
        ctx.set_particles(xyz)
        ctx.build_cells()
        one = ctx.local_matvec(np.ones((n, 3)))[0, 0]
        few, bounds = _launches(ctx, 4)
        many, again = _launches(ctx, 512)
        assert bounds == again
        # one eigenvalue, from sums of up to 3 n products of rounded vectors
        assert abs(bounds[0] - one) <= 1e-12 * one and abs(bounds[1] - one) <= 1e-12 * one
        # the steps that were under way when the end was seen, not 512 of ~10
        assert many <= 100


def test_two_beads():
    """six eigenvalues, two of them distinct per axis of the pair: the
    recurrence ends by the sixth step and finds both extremes"""
    xyz = np.array([[10.0, 10.0, 10.0], [12.5, 10.0, 10.0]])
    with G.Context(box_hi=(30.0,) * 3, precision=G.FP64) as ctx:
        ctx.set_particles(xyz)
        ctx.build_cells()
        m = np.stack([ctx.local_matvec(e.reshape(2, 3)).reshape(-1) for e in np.eye(6)])
        lam = np.linalg.eigvalsh(0.5 * (m + m.T))
        lo, hi = ctx.lanczos_bounds(k=6, seed=5)
        assert abs(lo - lam[0]) <= 1e-12 * lam[-1] and abs(hi - lam[-1]) <= 1e-12 * lam[-1]
