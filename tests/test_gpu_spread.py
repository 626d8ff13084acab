"""The element spread (every quadrature point of every element, reference
mode) through the C ABI against the FP64 oracle's per-point spread over
the element neighbour lists (assemble_stokes.C:645-662 with
ggem_stokes.C:117-128).

Tolerances: FP64 within 1e-12 (norm-wise); the FP32 path's error is
printed per component and bounded at 1e-6 norm-wise and 1e-5 of the
largest component.
"""
import numpy as np
import pytest

import ggem_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-12
ALPHA = 0.5


@pytest.fixture(scope="module", autouse=True)
def _built():
    from ggem_gb300 import build as B
    B.build()
    O.build_oracle(with_ref=False)


def rel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b))


def gauss_points(lo, L, nm):
    """2 x 2 x 2 Gauss points of every element of an nm[0] x nm[1] x nm[2]
    mesh (x fastest), element-major"""
    lo, L, nm = np.asarray(lo, float), np.asarray(L, float), np.asarray(nm)
    h = L / nm
    g = np.array([0.5 - 0.5 / np.sqrt(3.0), 0.5 + 0.5 / np.sqrt(3.0)])
    loc = np.array([[g[a], g[b], g[c]] for c in range(2) for b in range(2) for a in range(2)])
    ez, ey, ex = np.meshgrid(np.arange(nm[2]), np.arange(nm[1]), np.arange(nm[0]), indexing="ij")
    base = np.stack([ex.ravel(), ey.ravel(), ez.ravel()], axis=1)
    q = (base[:, None, :] + loc[None, :, :]) * h + lo
    return q.reshape(-1, 3), len(loc)


def _check(lo, L, nm, periodic, xyz, seed):
    lo, L = np.asarray(lo, float), np.asarray(L, float)
    hi = lo + L
    h = L / np.asarray(nm)
    sre = 0.5 * h.max() + 4.0 / ALPHA + 1e-3
    box = O.make_box(lo, hi, periodic)
    mesh = O.make_mesh(*nm, sre)
    c = O.constants(alpha=ALPHA)
    enb, _ = O.elem_lists(box, mesh, xyz)
    q, nq = gauss_points(lo, L, nm)
    qe = np.repeat(np.arange(int(np.prod(nm))), nq).astype(np.int32)
    f = np.random.default_rng(seed).standard_normal((len(xyz), 3))
    want = O.spread_qp(c, box, enb, xyz, f, q, qe)
    out = {}
    with G.Context(alpha=ALPHA, box_lo=tuple(lo), box_hi=tuple(hi), periodic=periodic,
                   nb_mode=G.NB_REFERENCE, n_mesh=tuple(nm), search_radius_e=sre,
                   precision=G.FP64) as ctx:
        ctx.set_particles(xyz)
        ctx.build_cells()
        ctx.set_quadrature(q, nq)
        for prec in (G.FP64, G.FP32):
            out[prec] = ctx.spread_elements(f, prec)
            again = ctx.spread_elements(f, prec)
            assert np.array_equal(out[prec], again)  # no state carried between calls
    e64 = rel(out[G.FP64], want)
    e32 = rel(out[G.FP32], want)
    comp = np.abs(out[G.FP32] - want).max() / np.abs(want).max()
    print(f"spread nm={nm} n={len(xyz)} periodic={periodic}: FP64 {e64:.2e}, FP32 norm-wise "
          f"{e32:.2e}, max component {comp:.2e} of the largest")
    assert e64 <= FP64_TOL
    assert e32 <= 1e-6 and comp <= 1e-5


def test_spread_small_mesh_whole_axis_stencil():
    """6 elements per axis: the element stencil covers every axis (offsets
    wrap, minimum image inside the brick)"""
    rng = np.random.default_rng(8)
    L = 24.0
    _check((0, 0, 0), (L,) * 3, (6, 6, 6), (1, 1, 1), rng.uniform(0, L, (150, 3)), 1)


def test_spread_fine_mesh_suspension():
    """h = 1.43 (the spread's mesh size), beads at phi = 0.1: bricks whose
    dilated frame wraps the periodic box faces"""
    xyz, L = G.make_suspension(44, 1500, 0.1)
    nm = int(np.floor(L / 1.414))
    _check((0, 0, 0), (L,) * 3, (nm,) * 3, (1, 1, 1), xyz, 2)


def test_spread_open_axis_offset_box():
    """a non-periodic z axis and a box away from the origin"""
    rng = np.random.default_rng(3)
    lo, L, nm = (-11.0, 5.0, 100.0), (36.0, 30.0, 24.0), (24, 20, 16)
    xyz = np.asarray(lo) + rng.uniform(0, 1, (1200, 3)) * np.asarray(L)
    _check(lo, L, nm, (1, 1, 0), xyz, 3)


def test_spread_dense_staging_in_several_passes():
    """more particles in a brick's dilated region than one shared-memory
    pass holds (512 FP32 / 256 FP64 records): the passes add up"""
    rng = np.random.default_rng(4)
    L = 40.0
    xyz = rng.uniform(0, L, (6400, 3))
    _check((0, 0, 0), (L,) * 3, (28, 28, 28), (1, 1, 1), xyz, 4)


def test_spread_wide_stencil_compact_bitmap():
    """elements of h = 0.55 under the spread's search radius (0.5 h + 8):
    offsets up to 15 elements, so the stencil (31 per axis) plus twice the
    2-element brick exceeds 32 and the kernel reads the compact stencil
    bitmap instead of the padded one (an open box, whose frames are clipped
    to the mesh, keeps the case small)"""
    rng = np.random.default_rng(6)
    L = 12 * 0.55
    _check((0, 0, 0), (L,) * 3, (12, 12, 12), (0, 0, 0), rng.uniform(0, L, (60, 3)), 5)


@pytest.mark.parametrize("prec", [G.FP64, G.FP32])
def test_spread_writes_zeros_where_no_particle_reaches(prec):
    """one bead in the corner of a wide mesh: the points out of its reach get
    0, whatever the output held before"""
    import torch
    nm, h = 40, 1.4
    L = nm * h
    q, nq = gauss_points((0, 0, 0), (L,) * 3, (nm,) * 3)
    with G.Context(alpha=ALPHA, box_hi=(L,) * 3, periodic=(0, 0, 0), nb_mode=G.NB_REFERENCE,
                   n_mesh=(nm,) * 3, search_radius_e=0.5 * h + 8.0 + 1e-3,
                   precision=G.FP64) as ctx:
        ctx.set_particles(np.array([[0.7, 0.7, 0.7]]))
        ctx.build_cells()
        ctx.set_quadrature(q, nq)
        f = torch.ones(3, dtype=torch.float64, device="cuda")
        rho = torch.full((len(q), 3), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        ctx.spread_elements_dev(f.data_ptr(), rho.data_ptr(), prec)
        ctx.synchronize()
        rho = rho.cpu().numpy()
    assert np.all(rho[np.abs(q).max(axis=1) > 0.7 + 8.7 + 2 * h] == 0.0)
    assert np.all(np.isfinite(rho)) and rho.max() > 0.0


def _grid_points(lo, L, nm, p, order):
    """p[0] x p[1] x p[2] points per element; order: which axis index runs
    fastest first"""
    h = np.asarray(L, float) / np.asarray(nm)
    g = [0.5 + 0.4 * np.linspace(-1.0, 1.0, k) if k > 1 else np.array([0.37]) for k in p]
    loc = []
    for idx in np.ndindex(*[p[d] for d in order[::-1]]):
        i = dict(zip(order[::-1], idx))
        loc.append([g[d][i[d]] for d in range(3)])
    ez, ey, ex = np.meshgrid(np.arange(nm[2]), np.arange(nm[1]), np.arange(nm[0]), indexing="ij")
    base = np.stack([ex.ravel(), ey.ravel(), ez.ravel()], axis=1)
    q = (base[:, None, :] + np.array(loc)[None, :, :]) * h + np.asarray(lo, float)
    return q.reshape(-1, 3), len(loc)


@pytest.mark.parametrize("p,order,nm,periodic,jitter", [
    ((2, 2, 2), (0, 1, 2), (21, 18, 17), (1, 1, 1), 0.0),   # frames inside the axes
    ((2, 2, 2), (2, 1, 0), (13, 6, 21), (1, 1, 0), 0.0),    # an axis shorter than the stencil
    ((3, 3, 3), (0, 1, 2), (18, 10, 5), (0, 1, 0), 0.0),    # three of 32 lanes idle
    ((1, 1, 1), (0, 1, 2), (19, 21, 3), (1, 0, 1), 0.0),    # 32 elements per warp
    ((3, 1, 2), (1, 2, 0), (7, 19, 18), (1, 1, 1), 0.0),    # uneven rule, partial bricks
    ((1, 16, 2), (1, 0, 2), (9, 5, 6), (0, 0, 0), 0.0),     # 32 points in 32 rows
    ((32, 1, 1), (0, 1, 2), (5, 4, 6), (0, 0, 0), 0.0),     # summed per pair: 32 along x
    ((2, 2, 2), (0, 1, 2), (17, 18, 19), (1, 1, 1), 1e-13),  # summed per pair: no grid
])
def test_spread_tensor_grid_matches_oracle(p, order, nm, periodic, jitter):
    """the separable sum of a tensor grid of points (and where the points are
    not one, the sum per pair) against the oracle; several bricks hold more
    members than one pass stages"""
    lo = np.array([-2.0, 3.0, 0.5])
    L = np.asarray(nm) * np.array([1.41, 1.3, 1.37])
    rng = np.random.default_rng(sum(p) + nm[0])
    n = 500
    xyz = lo + rng.uniform(0, 1, (n, 3)) * L
    xyz[:260] = lo + 0.3 * L * rng.uniform(0, 1, (260, 3)) + 0.2 * L  # a crowded corner
    q, nq = _grid_points(lo, L, nm, p, order)
    q = q + jitter * rng.standard_normal(q.shape)
    f = rng.standard_normal((n, 3))
    sre = 0.5 * 1.41 + 8.0 + 1e-3
    box, mesh = O.make_box(lo, lo + L, periodic), O.make_mesh(*nm, sre)
    enb, _ = O.elem_lists(box, mesh, xyz)
    qe = np.repeat(np.arange(int(np.prod(nm))), nq).astype(np.int32)
    want = O.spread_qp(O.constants(alpha=ALPHA), box, enb, xyz, f, q, qe)
    with G.Context(alpha=ALPHA, box_lo=tuple(lo), box_hi=tuple(lo + L), periodic=periodic,
                   nb_mode=G.NB_REFERENCE, n_mesh=nm, search_radius_e=sre,
                   precision=G.FP64) as ctx:
        ctx.set_particles(xyz)
        ctx.build_cells()
        ctx.set_quadrature(q, nq)
        got = ctx.spread_elements(f, G.FP64)
        assert np.array_equal(got, ctx.spread_elements(f, G.FP64))
    # ~60 terms per point, each within a few ulp of e^{-alpha^2 r^2} at
    # alpha^2 r^2 <= 25: 25 * 2^-52 per term, well below 1e-13 of the norm
    assert rel(got, want) <= 1e-13


@pytest.mark.parametrize("p", [(1, 1, 1), (3, 1, 1), (5, 1, 1), (2, 2, 2), (3, 3, 3)])
@pytest.mark.parametrize("members", [1, 3, 4, 28, 29, 31, 32, 33, 63, 64, 65, 97])
def test_fp32_spread_member_batches(p, members):
    """members per element around the batches of 32, the four lanes of a
    point and their blocks of eight, for one to 27 points per element, on
    the padded bitmap: a cluster that every element in reach lists whole,
    against the FP64 spread (1e-6 norm-wise, as above)"""
    nm, h = 24, 1.4
    L = nm * h
    rng = np.random.default_rng(members)
    xyz = 11.2 + rng.uniform(0.1, 1.3, (members, 3))
    f = rng.standard_normal((members, 3))
    q, nq = _grid_points((0, 0, 0), (L,) * 3, (nm,) * 3, p, (0, 1, 2))
    with G.Context(alpha=ALPHA, box_hi=(L,) * 3, nb_mode=G.NB_REFERENCE, n_mesh=(nm,) * 3,
                   search_radius_e=0.5 * h + 8.0 + 1e-3, precision=G.FP64) as ctx:
        ctx.set_particles(xyz)
        ctx.build_cells()
        ctx.set_quadrature(q, nq)
        want, got = ctx.spread_elements(f, G.FP64), ctx.spread_elements(f, G.FP32)
    assert rel(got, want) <= 1e-6


@pytest.mark.parametrize("p", [(2, 1, 1), (3, 3, 1), (4, 2, 2)])
@pytest.mark.parametrize("members", [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 48, 64, 65, 130])
@pytest.mark.parametrize("nm", [24, 11])
def test_fp32_spread_lanes_per_point(p, members, nm):
    """16 and 2 lanes per point around their pairs of members, blocks of eight
    and batches, on the padded bitmap and on a mesh that the stencil spans,
    against the FP64 spread (1e-6 norm-wise, as above)"""
    h = 1.4
    L = nm * h
    rng = np.random.default_rng(members)
    xyz = 5.6 + rng.uniform(0.1, 1.3, (members, 3))
    f = rng.standard_normal((members, 3))
    q, nq = _grid_points((0, 0, 0), (L,) * 3, (nm,) * 3, p, (0, 1, 2))
    with G.Context(alpha=ALPHA, box_hi=(L,) * 3, nb_mode=G.NB_REFERENCE, n_mesh=(nm,) * 3,
                   search_radius_e=0.5 * h + 8.0 + 1e-3, precision=G.FP64) as ctx:
        ctx.set_particles(xyz)
        ctx.build_cells()
        ctx.set_quadrature(q, nq)
        want, got = ctx.spread_elements(f, G.FP64), ctx.spread_elements(f, G.FP32)
        assert np.array_equal(got, ctx.spread_elements(f, G.FP32))
    assert rel(got, want) <= 1e-6


@pytest.mark.parametrize("prec", [G.FP64, G.FP32])
def test_captured_spread_follows_rebuilds(prec):
    """a caller's graph of the spread reads the context's stencil bitmap,
    which was sent up before, and the cells of the configuration at replay"""
    import torch
    nm, h, n = 20, 1.4, 700
    L = nm * h
    rng = np.random.default_rng(8)
    q, nq = _grid_points((0, 0, 0), (L,) * 3, (nm,) * 3, (2, 2, 2), (0, 1, 2))
    f = torch.from_numpy(rng.standard_normal((n, 3))).cuda()
    rho = torch.zeros((len(q), 3), dtype=torch.float64, device="cuda")
    st = torch.cuda.Stream()
    with G.Context(alpha=ALPHA, box_hi=(L,) * 3, nb_mode=G.NB_REFERENCE, n_mesh=(nm,) * 3,
                   search_radius_e=0.5 * h + 8.0 + 1e-3, precision=G.FP64) as ctx:
        ctx.set_stream(st.cuda_stream)
        torch.cuda.synchronize()
        ctx.set_particles(rng.uniform(0, L, (n, 3)))
        ctx.build_cells()
        ctx.set_quadrature(q, nq)
        ctx.spread_elements_dev(f.data_ptr(), rho.data_ptr(), prec)
        ctx.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            ctx.spread_elements_dev(f.data_ptr(), rho.data_ptr(), prec)
        for _ in range(2):
            ctx.set_particles(rng.uniform(0, L, (n, 3)))
            ctx.build_cells()
            ctx.spread_elements_dev(f.data_ptr(), rho.data_ptr(), prec)
            ctx.synchronize()
            live = rho.clone()
            rho.zero_()
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(rho, live) and float(live.abs().max()) > 0.0
        ctx.set_stream(0)
