"""The FP64 Chebyshev series of one right-hand side as one launch, in each of
its shapes, against the same series as single launches (which the kernel timer
selects) and against the oracle: the sizes where the lanes per target and the
targets per lane group change, ragged last blocks, rows longer than the cached
entries, element lists, every check interval, and series that end unconverged.

The two forms add the same terms in another order: y differs by a few ulp of
each of up to 30 terms of size <= |c_k| |x_k|, 1e-12 norm-wise; err1 is the
root of a difference of sums that agree to its square, 1e-6 for err1 >= 1e-3,
so 1e-15 of the sums is 1e-9 of it; 1e-6 leaves room for smaller ones."""
import numpy as np
import pytest

import ggem_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.fixture(scope="module", autouse=True)
def _built():
    from ggem_gb300 import build as B
    B.build()
    O.build_oracle(with_ref=False)


def rel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b))


def _suspension(n, phi=0.05):
    xyz, L = G.make_suspension(n % 1000 + 1, n, phi)
    return xyz, max(L, 21.5)


def _contexts(**params):
    one, many = (G.Context(precision=G.FP64, **params) for _ in range(2))
    many.set_kernel_timing(True)  # single launches
    return one, many


def _compare(one, many, xyz, checks=(1, 0, 3), N=30, tol=1e-3, bounds=None):
    n = len(xyz)
    xi = np.random.default_rng(n).standard_normal((n, 3))
    for c in (one, many):
        c.set_particles(xyz)
        c.build_cells()
    lo, hi = bounds or one.lanczos_bounds(k=24, seed=7)
    lo, hi = lo / 1.05, hi * 1.05
    for ce in checks:
        for _ in range(2):  # (an adaptive series starts where the last one ended)
            a, b = one.launch_count(), many.launch_count()
            y1, r1 = one.cheb_inv_sqrt(xi, N, lo, hi, tol, check_every=ce)
            y2, r2 = many.cheb_inv_sqrt(xi, N, lo, hi, tol, check_every=ce)
            assert one.launch_count() - a < many.launch_count() - b or N == 1
            for k in ("converged", "n_terms", "n_matvecs"):
                assert r1[0][k] == r2[0][k], (ce, k, r1, r2)
            for k in ("err1", "err2"):
                assert r1[0][k] == pytest.approx(r2[0][k], rel=1e-6, abs=1e-9), (ce, k)
            assert rel(y1, y2) <= TOL, ce
            rc1, dw1, _ = one.brownian_displacement(xi, N, lo, hi, tol, check_every=ce)
            rc2, dw2, _ = many.brownian_displacement(xi, N, lo, hi, tol, check_every=ce)
            assert rc1 == rc2 == (0 if r1[0]["converged"] else G.ERR_CHEB_NOT_CONVERGED)
            if rc1 == 0:
                assert rel(dw1, dw2) <= TOL, ce
    return lo, hi, xi


# 3648 targets fill <16, 4> on 152 SMs, 17024 one round of <8, 0>; from 80000
# on <4, 0> takes 34048 a round
@pytest.mark.parametrize("n", [2, 7, 9, 1000, 3647, 3648, 3649, 17024, 17025, 20011, 79999, 80000,
                               80033])
def test_shapes_and_rounds(n):
    xyz, L = _suspension(n)
    one, many = _contexts(box_hi=(L,) * 3)
    with one, many:
        _compare(one, many, xyz, checks=(1, 0, 3) if n < 30000 else (1, 0))


@pytest.mark.parametrize("n", [1500, 5000])
def test_against_the_oracle(n):
    xyz, L = _suspension(n)
    one, many = _contexts(box_hi=(L,) * 3)
    with one, many:
        lo, hi, xi = _compare(one, many, xyz, checks=(1,))
        box = O.make_box([0] * 3, [L] * 3, [1, 1, 1])
        nb = O.neighbors_cutoff(box, xyz, 7.0)
        op = O.Operator(matvec=(O.constants(alpha=0.5), box, xyz, nb, O.SELF_BEAD, 8))
        want, rep = O.cheb_inv_sqrt(op, xi.reshape(-1), 30, lo, hi, 1e-3)
        got, mine = one.cheb_inv_sqrt(xi, 30, lo, hi, 1e-3, check_every=1)
        assert mine[0]["n_terms"] == rep.n_terms and mine[0]["converged"] == rep.converged
        assert rel(got.reshape(-1), want) <= TOL


@pytest.mark.parametrize("n", [900, 3648, 3700])
def test_rows_longer_than_the_cached_entries(n):
    """a crowded box: rows of 60 to 400 entries, uneven between the targets"""
    L = 24.0
    rng = np.random.default_rng(n)
    xyz = rng.uniform(0.0, L, (n, 3))
    xyz[: n // 3] *= 0.5
    one, many = _contexts(box_hi=(L,) * 3, br0=0.5)
    with one, many:
        _compare(one, many, xyz, bounds=(0.02, 30.0))


@pytest.mark.parametrize("n", [60, 2500, 5000])
def test_element_lists(n):
    xyz, L = _suspension(n)
    nm = int(np.ceil(L / 1.414))
    one, many = _contexts(box_hi=(L,) * 3, nb_mode=G.NB_REFERENCE, n_mesh=(nm,) * 3,
                          search_radius_e=0.5 * L / nm + 8.0 + 1e-3)
    with one, many:
        _compare(one, many, xyz)


@pytest.mark.parametrize("N", [1, 2, 3, 5, 9, 50])
@pytest.mark.parametrize("tol", [1e-3, 1e-14])
def test_degrees_and_series_that_end_unconverged(N, tol):
    xyz, L = _suspension(1200)
    one, many = _contexts(box_hi=(L,) * 3)
    with one, many:
        _compare(one, many, xyz, checks=(1, 0, 2, 4), N=N, tol=tol)


@pytest.mark.parametrize("point", [G.LAGRANGIAN_POINT, G.POINT_PARTICLE])
def test_other_self_terms(point):
    xyz, L = _suspension(1200)
    one, many = _contexts(box_hi=(L,) * 3, point_type=point)
    with one, many:
        _compare(one, many, xyz, checks=(1, 0), bounds=(0.2, 8.0))


def test_result_over_the_noise():
    """the displacement may be written over its noise vector"""
    import torch
    xyz, L = _suspension(4000)
    xi = torch.from_numpy(np.random.default_rng(1).standard_normal((4000, 3))).cuda()
    dw = torch.empty_like(xi)
    with G.Context(precision=G.FP64, box_hi=(L,) * 3) as ctx:
        ctx.set_particles(xyz)
        ctx.build_cells()
        lo, hi = ctx.lanczos_bounds(k=24, seed=7)
        torch.cuda.synchronize()
        args = (1, 30, lo / 1.05, hi * 1.05, 1e-3)
        assert ctx.brownian_displacement_dev(xi.data_ptr(), dw.data_ptr(), *args)[0] == 0
        ctx.synchronize()
        assert ctx.brownian_displacement_dev(xi.data_ptr(), xi.data_ptr(), *args)[0] == 0
        ctx.synchronize()
        assert torch.equal(xi, dw)


@pytest.mark.parametrize("n", [3000, 20000, 90000])
def test_wait_that_runs_out(n):
    """with one poll per wait the blocks give up, the call reports the timeout
    and the next series is exact.  (Every wait is bounded: the kernel ends as
    soon as one block has given up.)"""
    xyz, L = _suspension(n)
    xi = np.random.default_rng(2).standard_normal((n, 3))
    with G.Context(precision=G.FP64, box_hi=(L,) * 3) as ctx:
        ctx.set_particles(xyz)
        ctx.build_cells()
        lo, hi = ctx.lanczos_bounds(k=24, seed=7)
        args = (xi, 30, lo / 1.05, hi * 1.05, 1e-3)
        want, _ = ctx.cheb_inv_sqrt(*args)
        ctx.set_series_polls(1)
        with pytest.raises(G.GGEMError) as e:
            ctx.cheb_inv_sqrt(*args)
        assert e.value.code == G.ERR_TIMEOUT
        ctx.set_series_polls(0)
        got, rep = ctx.cheb_inv_sqrt(*args)
        assert rep[0]["converged"] and np.array_equal(got, want)
