"""FP32 pair-list rows where the builder's loops have their edges: targets per
cell around its groups of two and four and its chunks of 32, candidates around
its rounds of 256 and its queue, stencils of one and of several chunks of 32
cells, and the half list beside the full one.  Lists are whole numbers: equal
to the oracle's."""
import numpy as np
import pytest

import ggem_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from ggem_gb300 import build as B
    B.build()
    O.build_oracle(with_ref=False)


@pytest.mark.parametrize("cell_div", [1, 2])
@pytest.mark.parametrize("inner,outer", [(1, 0), (1, 40), (2, 160), (3, 161), (4, 190), (5, 220),
                                         (6, 255), (7, 256), (31, 257), (32, 300), (33, 500),
                                         (67, 900)])
def test_rows_match_oracle(inner, outer, cell_div):
    L = 28.0
    rng = np.random.default_rng(1000 * inner + outer)
    # `inner` beads in one cell's corner, `outer` within reach around it, a few far away
    xyz = np.concatenate([rng.uniform(14.1, 17.4, (inner, 3)), rng.uniform(7.5, 24.0, (outer, 3)),
                          rng.uniform(0.0, L, (5, 3))])
    nb = O.neighbors_cutoff(O.make_box([0] * 3, [L] * 3, [1, 1, 1]), xyz, 7.0)
    f = rng.standard_normal(xyz.shape)
    for half in (False, True):
        with G.Context(box_hi=(L,) * 3, rc=7.0, cell_div=cell_div) as ctx:
            ctx.set_symmetric_pairs(half)
            for _ in range(2):  # the second build has its row width
                ctx.set_particles(xyz)
                ctx.build_cells()
            off, ids = ctx.neighbors()
            assert np.array_equal(off, nb.offsets) and np.array_equal(ids, nb.ids)
            assert ctx.pair_count() == nb.offsets[-1]
            u = ctx.local_matvec(f, G.SELF_BEAD)
            if not half:
                full = u
            # each unordered pair once: the same operator as with the full list (FP32 sums of
            # up to ~970 terms in blocks, 6e-8 each: 1e-5 norm-wise)
            assert np.linalg.norm(u - full) <= 1e-5 * np.linalg.norm(full)


@pytest.mark.parametrize("nc", [(3, 3, 3), (16, 16, 16), (17, 16, 16), (24, 24, 24), (32, 32, 32),
                                (33, 32, 32), (64, 64, 32), (65, 64, 32)])
def test_cell_offsets_over_scan_blocks(nc):
    """cell counts around the scan's tiles of 4096, its two to eight blocks
    and its limit of 131072: lists equal to the oracle's, twice (the first
    build leaves its counters for the second)"""
    L = 7.0 * np.asarray(nc) + 1.0
    rng = np.random.default_rng(int(np.prod(nc)))
    box = O.make_box([0] * 3, list(L), [1, 1, 1])
    with G.Context(box_hi=tuple(L), rc=7.0) as ctx:
        for k in range(2):
            n = (4000, 2500)[k]
            # half of the beads in a slab, so that some rows have entries
            xyz = rng.uniform(0.0, 1.0, (n, 3)) * L
            xyz[::2, 2] = 0.6 * L[2] + 3.0 * xyz[::2, 2] / L[2]
            nb = O.neighbors_cutoff(box, xyz, 7.0)
            ctx.set_particles(xyz)
            ctx.build_cells()
            off, ids = ctx.neighbors()
            assert np.array_equal(off, nb.offsets) and np.array_equal(ids, nb.ids)
