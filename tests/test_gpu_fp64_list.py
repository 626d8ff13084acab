"""The FP64 operator over its own pair list (the default of FP64 contexts):
cut-off and element lists against the oracle and against the cell sweep, at
the sizes where the lanes per target change, on meshes whose stencil wraps or
spans an axis, for splitting parameters that move the tensor's pieces, and
under stream capture.

Both sides sum ~100 terms per component with a few ulp each (1e-16 relative
to the largest): 1e-13 norm-wise leaves a factor of ten over 100 ulp."""
import numpy as np
import pytest

import ggem_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-13


@pytest.fixture(scope="module", autouse=True)
def _built():
    from ggem_gb300 import build as B
    B.build()
    O.build_oracle(with_ref=False)


def rel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b))


def _apply(ctx, xyz, f):
    ctx.set_particles(xyz)
    ctx.build_cells()
    return ctx.local_matvec(f, G.SELF_BEAD)


@pytest.mark.parametrize("n,nrhs", [(1, 1), (2, 3), (300, 1), (300, 7), (2499, 1), (2500, 1),
                                    (79999, 1), (80000, 2)])
def test_cutoff_list_matches_oracle_and_sweep(n, nrhs):
    L = 40.0 if n < 300 else (n / 0.02) ** (1.0 / 3.0)
    rng = np.random.default_rng(n)
    xyz = rng.uniform(0.0, L, (n, 3))
    f = rng.standard_normal((nrhs, n, 3))
    box = O.make_box([0] * 3, [L] * 3, [1, 1, 1])
    nb = O.neighbors_cutoff(box, xyz, 7.0)
    c = O.constants(alpha=0.5)
    with G.Context(box_hi=(L,) * 3, precision=G.FP64) as ctx, \
            G.Context(box_hi=(L,) * 3, precision=G.FP64) as swept:
        swept.set_fp64_pair_list(False)
        for _ in range(2):  # the list comes with the matvec, then with the build
            got = _apply(ctx, xyz, f)
            for r in range(nrhs):
                assert rel(got[r], O.local_matvec(c, box, xyz, nb, f[r], O.SELF_BEAD)) <= TOL
        assert rel(got, _apply(swept, xyz, f)) <= TOL


@pytest.mark.parametrize("alpha,br0", [(0.1, 1.0), (0.5, 0.25), (0.25, 2.0)])
def test_tensor_pieces_over_splitting_parameters(alpha, br0):
    rc = 4.0 / alpha
    L, n = 3.2 * rc, 400
    rng = np.random.default_rng(5)
    # pairs over every octave of r, down to the r < 1e-6 branch
    xyz = rng.uniform(0.0, L, (n, 3))
    for k in range(40):
        xyz[2 * k + 1] = xyz[2 * k] + 10.0 ** (-7 + 0.2 * k) * np.array([0.6, -0.64, 0.48])
    xyz %= L
    f = rng.standard_normal((n, 3))
    box = O.make_box([0] * 3, [L] * 3, [1, 1, 1])
    c = O.constants(alpha=alpha, br0=br0)
    want = O.local_matvec(c, box, xyz, O.neighbors_cutoff(box, xyz, rc), f, O.SELF_BEAD)
    with G.Context(alpha=alpha, br0=br0, box_hi=(L,) * 3, rc=rc, precision=G.FP64) as ctx:
        assert rel(_apply(ctx, xyz, f), want) <= 1e-12


@pytest.mark.parametrize("nm,periodic", [((13, 12, 14), (1, 1, 1)), ((40, 22, 21), (1, 1, 1)),
                                         ((30, 24, 9), (0, 1, 0)), ((6, 5, 7), (1, 0, 1)),
                                         ((1, 3, 40), (1, 1, 0))])
def test_element_lists_match_oracle(nm, periodic):
    h = np.array([1.4, 1.3, 1.37])
    lo, L = np.array([-3.0, 0.5, 2.0]), np.asarray(nm) * h
    n = 700
    rng = np.random.default_rng(sum(nm))
    xyz = lo + rng.uniform(0.0, 1.0, (n, 3)) * L
    f = rng.standard_normal((n, 3))
    sre = 0.5 * h.max() + 8.0 + 1e-3
    box = O.make_box(lo, lo + L, periodic)
    mesh = O.make_mesh(*nm, sre)
    nb = O.neighbors_reference(box, mesh, xyz)
    want = O.local_matvec(O.constants(alpha=0.5), box, xyz, nb, f, O.SELF_BEAD)
    with G.Context(box_lo=tuple(lo), box_hi=tuple(lo + L), periodic=periodic,
                   nb_mode=G.NB_REFERENCE, n_mesh=nm, search_radius_e=sre,
                   precision=G.FP64) as ctx:
        for _ in range(2):
            assert rel(_apply(ctx, xyz, f), want) <= 1e-12


def test_captured_matvec_follows_rebuilds():
    """a caller's graph of the FP64 matvec stays valid when the particles and
    with them the width of the list's rows change"""
    import torch
    n, L = 600, 40.0
    rng = np.random.default_rng(3)
    spread = rng.uniform(0.0, L, (n, 3))
    crowded = rng.uniform(0.0, 6.0, (n, 3))
    f = torch.from_numpy(rng.standard_normal((n, 3))).cuda()
    u = torch.zeros_like(f)
    st = torch.cuda.Stream()
    with G.Context(box_hi=(L,) * 3, precision=G.FP64) as ctx:
        ctx.set_stream(st.cuda_stream)
        torch.cuda.synchronize()
        ctx.set_particles(spread)
        ctx.build_cells()
        ctx.local_matvec_dev(f.data_ptr(), u.data_ptr())
        ctx.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            ctx.local_matvec_dev(f.data_ptr(), u.data_ptr())
        for xyz in (crowded, spread):
            ctx.set_particles(xyz)
            ctx.build_cells()
            ctx.local_matvec_dev(f.data_ptr(), u.data_ptr())
            ctx.synchronize()
            live = u.clone()
            u.zero_()
            g.replay()
            torch.cuda.synchronize()
            assert rel(u.cpu().numpy(), live.cpu().numpy()) <= TOL
        ctx.set_stream(0)


def _tensor_a(alpha, ksi, k, r):
    """A(r) to 60 digits: k [(erf(ksi r) - erf(alpha r)) / r + 2 / sqrt(pi)
    (ksi e^{-(ksi r)^2} - alpha e^{-(alpha r)^2})] with the erf by their series"""
    from decimal import Decimal as D, getcontext
    getcontext().prec = 110
    pi = D("3.14159265358979323846264338327950288419716939937510582097494459230781640628620899862803")

    def half_erf(x):  # sqrt(pi) / 2 erf(x); 1 - erf(12) < 1e-62
        if x > 12:
            return pi.sqrt() / 2
        t, s, n = x, x, 0
        while abs(t) > D(10) ** -70:
            n += 1
            t *= -x * x / n
            s += t / (2 * n + 1)
        return s

    a, q, r = D(float(alpha)), D(float(ksi)), D(float(r))
    c = 2 / pi.sqrt()
    c1 = c * (half_erf(q * r) - half_erf(a * r)) / r
    c2 = c * (q * (-(q * r) ** 2).exp() - a * (-(a * r) ** 2).exp())
    return D(float(k)) * (c1 + c2)


@pytest.mark.parametrize("alpha,br0,rc", [(0.5, 1.0, 7.0), (0.1, 1.0, 35.0), (0.5, 0.25, 8.0),
                                          (0.01, 10.0, 0.5)])
def test_tensor_is_good_to_its_rounding(alpha, br0, rc):
    """A(r) of isolated pairs, from 1e-4 rc to rc, against 60 digits.  The
    value carries the rounding of its constant coefficient and of the last
    fused multiply-add, half an ulp or 2^-53 of A(0) at most each: 9e-17 rms;
    with the samples' own rounding averaged over 12 of them, 1.5e-16."""
    from decimal import Decimal as D
    m, g = 192, 6
    rng = np.random.default_rng(2)
    r = rc * np.concatenate([10.0 ** rng.uniform(-4, 0, m // 2), rng.uniform(0.02, 1.0, m // 2)])
    i = np.arange(m)
    base = (np.stack([i % g, (i // g) % g, i // (g * g)], 1) + 0.5) * 3.0 * rc
    other = base.copy()
    other[:, 0] += r * (1 - 1e-9)
    r = other[:, 0] - base[:, 0]  # exact
    f = np.zeros((2 * m, 3))
    f[:m, 1] = 1.0
    with G.Context(alpha=alpha, br0=br0, box_hi=(3.0 * rc * g,) * 3, periodic=(0, 0, 0), rc=rc,
                   precision=G.FP64) as ctx:
        ctx.set_particles(np.concatenate([base, other]))
        ctx.build_cells()
        got = ctx.local_matvec(f, G.SELF_NONE)[m:, 1]
        c = ctx.constants()
    a0 = c.one_eight_pi_mu * 4.0 / np.sqrt(np.pi) * (c.ksi - c.alpha)
    err = np.array([float(D(float(a)) - _tensor_a(c.alpha, c.ksi, c.one_eight_pi_mu, x)) / a0
                    for a, x in zip(got, r)])
    assert np.sqrt(np.mean(err ** 2)) <= 1.5e-16
