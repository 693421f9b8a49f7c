"""Near-field sums at the edges of the pair arithmetic: scales near the ends of the exponent range,
coincident bodies, leaf sizes around the lane tiles.  The reference is the plain all-pairs sum in
extended precision; the bound is the rounding of a sum of n terms of a few ulps each, relative to
the sum of the terms' magnitudes."""
import ctypes as C

import numpy as np
import pytest

import fastmultipole_b200 as fm
from fastmultipole_b200 import _lib as L

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def ctx():
    c = fm.Context(0)
    yield c
    c.close()


def bodies(n, kind, scale, seed):
    rng = np.random.default_rng(seed)
    b = np.zeros((n, 5 if kind == 1 else 7))
    b[:, :3] = (rng.random((n, 3)) - 0.3) * scale
    b[:, 4:] = rng.standard_normal((n, b.shape[1] - 4))
    return b


def sums(tp, b, hess):
    """(value, sum of |terms|) of potential, gradient / velocity, velocity gradient, extended precision."""
    x, s = b[:, :3].astype(np.longdouble), b[:, 4:].astype(np.longdouble)
    d = tp.astype(np.longdouble)[:, None, :] - x[None]
    r2 = (d * d).sum(-1)
    with np.errstate(divide="ignore", invalid="ignore"):
        w = np.where(r2 > 0, 1 / np.sqrt(np.where(r2 > 0, r2, 1)), 0)
    f = 1 / (4 * np.longdouble(np.pi))
    w3 = w ** 3
    if s.shape[1] == 1:
        t0, t1 = w * s[:, 0], d * (w3 * s[:, 0])[..., None]
        return [(f * t0.sum(1), f * abs(t0).sum(1)), (f * t1.sum(1), f * abs(t1).sum(1))]
    c = np.cross(np.broadcast_to(s[None], d.shape), d)
    mag = abs(s[None]) @ np.ones((3, 3)) * np.sqrt(r2)[..., None]  # bound of the two terms of a component
    out = [None, (f * (c * w3[..., None]).sum(1), f * (mag * w3[..., None]).sum(1))]
    if hess:
        eps = np.zeros((3, 3, 3))
        for i, j, k in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
            eps[i, j, k], eps[i, k, j] = 1, -1
        # du_j / dx_i = eps_jki G_k / r^3 - 3 d_i (G x d)_j / r^5, component 3 i + j
        t = np.einsum("jki,sk->sij", eps, s.astype(float))[None] * w3[..., None, None] \
            - 3 * d[..., :, None] * c[..., None, :] * (w3 * w * w)[..., None, None]
        m = 4 * (abs(s).sum(1)[None] * w3)[..., None, None] * np.ones((3, 3))
        out.append((f * t.sum(1).reshape(len(tp), 9), f * m.sum(1).reshape(len(tp), 9)))
    return out


@pytest.mark.parametrize("kind,hess", [(1, False), (3, False), (3, True)])
@pytest.mark.parametrize("scale", [1.0, 1e-40, 1e40, 1e55])
@pytest.mark.parametrize("leaf,n", [(7, 101), (30, 333), (200, 1)])
def test_f64_pairs(ctx, kind, hess, scale, leaf, n):
    b = bodies(n, kind, scale, 11)
    # targets: every third source (coincident pairs across the two trees) and other points
    tp = np.concatenate([b[::3, :3], bodies(40, kind, scale, 12)[:, :3]])
    for sep in (False, True):
        pos = tp if sep else b[:, :3]
        # no pair is well separated: the near field holds all pairs
        opt = fm.make_options(expansion_order=4, leaf_size_source=leaf, scalar_potential=kind == 1, hessian=hess,
                              farfield=False, multipole_acceptance=1e-9)
        out, res = fm.solve_buffers(b, kind, opt, pos if sep else None, ctx=ctx)
        for cols, ref in zip((slice(3, 4), slice(4, 7), slice(7, 16)), sums(pos, b, hess)):
            if ref is None:
                continue
            got = out[:, cols].reshape(np.shape(ref[0]))
            assert np.all(np.isfinite(got))
            assert np.all(abs(got - ref[0]) <= 4 * (n + 16) * EPS * ref[1] + 1e-300)


def test_f64_overflowing_gradient_keeps_the_potential(ctx):
    """1 / r^3 overflows, q / r does not: the potential is exact, as it is without the gradient."""
    b = bodies(80, 1, 1e-110, 5)
    opt = fm.make_options(expansion_order=3, leaf_size_source=20, scalar_potential=True, farfield=False,
                          multipole_acceptance=1e-9)
    out, _ = fm.solve_buffers(b, 1, opt, ctx=ctx)
    v, m = sums(b[:, :3], b, False)[0]
    assert np.all(abs(out[:, 3] - v) <= 4 * (80 + 16) * EPS * m)
    assert not np.all(np.isfinite(out[:, 4:7]))


@pytest.mark.parametrize("scale,strength", [(1e40, 1e-200), (1e3, 1e-300), (1.0, 1e-307), (1e40, 1e-160)])
@pytest.mark.parametrize("mix", [False, True])
def test_f64_potential_of_tiny_strengths(ctx, scale, strength, mix):
    """q / r is a normal number where q / r^3 is not: the potential keeps all its bits (mix: beside
    bodies of ordinary strength and of none)."""
    b = bodies(150, 1, scale, 7)
    b[:, 4] = (1 + abs(b[:, 4])) * strength
    if mix:
        b[::7, 4] = 0.0
        b[3::50, 4] *= 1e20
    v, m = sums(b[:, :3], b, False)[0]
    tol = 4 * (150 + 16) * EPS * m
    opt = fm.make_options(expansion_order=3, leaf_size_source=20, scalar_potential=True, farfield=False,
                          multipole_acceptance=1e-9)
    out, _ = fm.solve_buffers(b, 1, opt, ctx=ctx)
    assert np.all(abs(out[:, 3] - v) <= tol + 2.0 ** -1073)
    out = np.zeros((150, 16))
    src = L.SourceSystem(1, 150, 5, b.ctypes.data, L.FMM_MEMORY_HOST)
    tgt = L.TargetSystem(150, None, 0, out.ctypes.data, L.FMM_MEMORY_HOST)
    ctx.check(L.lib().fmm_direct(ctx.handle, C.byref(tgt), C.byref(src), 1, 1, 0, L.FMM_PRECISION_F64))
    assert np.all(abs(out[:, 3] - v) <= tol + 2.0 ** -1073)


@pytest.mark.parametrize("kind,hess", [(1, False), (3, False), (3, True)])
@pytest.mark.parametrize("leaf,ls_t", [(16, 3), (60, 47), (150, 20)])
def test_items_cover_every_pair(ctx, kind, hess, leaf, ls_t):
    """Enough pairs for the launch to be cut into items: rows of several target tiles, ragged tiles, and
    rows of a few targets with thousands of sources."""
    b = bodies(4111, kind, 1.0, 31)
    pos = np.concatenate([bodies(1100, kind, 0.2, 32)[:, :3], bodies(37, kind, 3.0, 33)[:, :3], b[:64, :3]])
    res = {}
    for prec in ("f64", "mixed"):
        opt = fm.make_options(expansion_order=3, leaf_size_source=leaf, leaf_size_target=ls_t,
                              scalar_potential=kind == 1, hessian=hess, farfield=False, multipole_acceptance=1e-9,
                              precision=prec)
        res[prec], _ = fm.solve_buffers(b, kind, opt, pos, ctx=ctx)
    for cols, ref in zip((slice(3, 4), slice(4, 7), slice(7, 16)), sums(pos, b, hess)):
        if ref is None:
            continue
        got = res["f64"][:, cols].reshape(np.shape(ref[0]))
        assert np.all(abs(got - ref[0]) <= 4 * (len(b) + 16) * EPS * ref[1])
        # FP32 coordinates relative to a target leaf: 2^-24 of its extent against the distances of a
        # few thousand bodies in a unit cube (about 1e-2), order 5
        mixed = res["mixed"][:, cols].reshape(np.shape(ref[0]))
        assert np.linalg.norm(mixed - got) <= 1e-4 * np.linalg.norm(got)


@pytest.mark.parametrize("kind,hess", [(1, False), (3, True)])
@pytest.mark.parametrize("leaf,ls_t", [(16, 3), (60, 47), (300, 150)])
def test_items_of_nested_rows(ctx, kind, hess, leaf, ls_t):
    """SelfTuning: target branches that are not leaves have rows too, of several tiles, and share their
    targets with the rows of their descendants."""
    b = bodies(8111, kind, 1.0, 35)
    pos = np.concatenate([bodies(3000, kind, 0.4, 36)[:, :3], bodies(201, kind, 3.0, 37)[:, :3]])
    some = np.arange(0, len(pos), 19)
    ref = sums(pos[some], b, hess)
    for prec, eps in (("f64", None), ("mixed", 1e-4)):
        opt = fm.make_options(expansion_order=3, leaf_size_source=leaf, leaf_size_target=ls_t, scalar_potential=kind == 1,
                              hessian=hess, farfield=False, multipole_acceptance=1e-9, precision=prec,
                              interaction_list_method=fm.SelfTuning())
        out, res = fm.solve_buffers(b, kind, opt, pos, ctx=ctx)
        assert res.n_p2p_pairs == len(b) * len(pos)
        for cols, r in zip((slice(3, 4), slice(4, 7), slice(7, 16)), ref):
            if r is None:
                continue
            got = out[some, cols].reshape(np.shape(r[0]))
            if eps is None:  # (rows of a branch and its ancestors: a few more additions)
                assert np.all(abs(got - r[0]) <= 4 * (len(b) + 32) * EPS * r[1])
            else:
                assert np.linalg.norm((got - r[0]).astype(float)) <= eps * np.linalg.norm(r[0].astype(float))
