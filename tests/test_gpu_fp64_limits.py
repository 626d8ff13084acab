"""FP64 contexts where the FP32 filter of the pair list cannot separate the
pairs at the cut-off: cells many times the cut-off (an axis of 2048 cells is
the largest), and cut-offs outside the FP32 range.  Every call gives what the
cell sweep gives, which compares FP64 distances.

Both sides sum a few terms per component: 1e-13 norm-wise."""
import numpy as np
import pytest

import ggem_gb300 as G

pytestmark = pytest.mark.gpu
TOL = 1e-13


@pytest.fixture(scope="module", autouse=True)
def _built():
    from ggem_gb300 import build as B
    B.build()


def rel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b))


def _both(xyz, f, **params):
    """u over the default context's own choice and over the cells"""
    out = []
    for swept in (False, True):
        with G.Context(precision=G.FP64, **params) as ctx:
            if swept:
                ctx.set_fp64_pair_list(False)
            for _ in range(2):  # a list comes with the matvec, then with the build
                ctx.set_particles(xyz)
                ctx.build_cells()
                u = ctx.local_matvec(f, G.SELF_BEAD)
            out.append(u)
    return out


@pytest.mark.parametrize("cells", [1.0, 64.0, 90.0, 2e4])
def test_pairs_at_the_cutoff_in_wide_cells(cells):
    """an axis of 2048 cells, each `cells` cut-offs long, and pairs at rc
    (1 + d) with d down to 1e-6 on both sides"""
    rc = 7.0
    L = (2048 * cells * rc, 30.0, 30.0)
    rng = np.random.default_rng(11)
    m = 400
    a = rng.uniform(0.0, 1.0, (m, 3)) * (np.asarray(L) - 20.0) + 10.0
    v = rng.standard_normal((m, 3))
    v *= (rc * (1.0 + rng.choice([-1.0, 1.0], m) * 10.0 ** rng.uniform(-6, -2.5, m))
          / np.linalg.norm(v, axis=1))[:, None]
    xyz = np.concatenate([a, a + v])
    f = rng.standard_normal(xyz.shape)
    # alpha small enough that the tensor at rc is far from rounding
    got, want = _both(xyz, f, box_hi=L, periodic=(0, 1, 1), rc=rc, alpha=0.1)
    assert rel(got, want) <= TOL


@pytest.mark.parametrize("rc,scale", [(1e6, 1.0), (1e20, 1.0), (1e200, 1.0), (1e-23, 1e-24), (7.0, 1.0)])
def test_cutoffs_outside_the_fp32_range(rc, scale):
    """an open box of 20 `scale`: every pair within the larger cut-offs"""
    rng = np.random.default_rng(3)
    n = 300
    xyz = rng.uniform(0.0, 20.0 * scale, (n, 3))
    f = rng.standard_normal((n, 3))
    got, want = _both(xyz, f, box_hi=(20.0 * scale,) * 3, periodic=(0, 0, 0), rc=rc)
    assert np.all(np.isfinite(want))
    assert rel(got, want) <= TOL


def test_rows_no_wider_than_the_particles():
    """a cut-off beyond an open box lists every pair: rows of n entries"""
    import torch
    n = 300
    rng = np.random.default_rng(4)
    xyz, f = rng.uniform(0.0, 20.0, (n, 3)), rng.standard_normal((n, 3))
    with G.Context(precision=G.FP64, box_hi=(20.0,) * 3, periodic=(0, 0, 0), rc=1e4) as ctx:
        ctx.set_particles(xyz)
        ctx.build_cells()
        free = torch.cuda.mem_get_info()[0]
        ctx.local_matvec(f, G.SELF_BEAD)
        assert free - torch.cuda.mem_get_info()[0] <= 64 << 20


def test_only_configurations_with_products_build_the_list():
    """after one product the builds that no product follows (a context that
    only spreads from then on) cost what they cost before it"""
    rng = np.random.default_rng(5)
    xyz, f = rng.uniform(0.0, 40.0, (500, 3)), rng.standard_normal((500, 3))
    with G.Context(precision=G.FP64, box_hi=(40.0,) * 3) as ctx:
        def launches(call):
            a = ctx.launch_count()
            call()
            return ctx.launch_count() - a

        ctx.set_particles(xyz)
        ctx.build_cells()
        fresh = launches(ctx.build_cells)
        ctx.local_matvec(f)
        ctx.build_cells()  # prepared for the product that usually follows
        assert launches(ctx.build_cells) == fresh
        # with a product on every configuration the list comes with the build
        for _ in range(3):
            ctx.local_matvec(f)
            ctx.build_cells()
            assert launches(lambda: ctx.local_matvec(f)) == 3  # order, product, order
