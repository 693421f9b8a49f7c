"""Translations of every instantiated order, plain and error-controlled, against the CPU restatement
of the reference: the orders around each kernel variant's limit, point sources and vortex particles."""
import numpy as np
import pytest

import fastmultipole_b200 as fm
from fastmultipole_b200 import _lib as L
import oracle_lib as O
from test_gpu_fmm import opt_pair

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = fm.Context(0)
    yield c
    c.close()


def bodies(n, kind, seed):
    rng = np.random.default_rng(seed)
    b = np.zeros((n, 5 if kind == 1 else 7))
    b[:, :3] = rng.random((n, 3)) ** 2
    b[:, 4:] = rng.standard_normal((n, b.shape[1] - 4)) / n
    return b


METHODS = [None, fm.PowerAbsoluteGradient, fm.PowerRelativeGradient, fm.RotatedCoefficientsAbsoluteGradient,
           fm.RotatedCoefficientsRelativeGradient, fm.PowerRelativePotential]


@pytest.mark.parametrize("kind", [1, 3])
@pytest.mark.parametrize("method", METHODS, ids=[m.__name__ if m else "plain" for m in METHODS])
@pytest.mark.parametrize("p", [1, 4, 5, 9, 12, 13, 16, 17, 20])
@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_orders_match_oracle(ctx, kind, method, p, precision):
    if precision == "mixed" and (method is None or (kind == 1 and p <= 12)):
        pytest.skip("FP32 translations, and FP64 ones already run: test_fp32_translations")
    n = 900
    b = bodies(n, kind, 3)
    tol = None if method is None else method(3e-6 if "Relative" in method.__name__ else 1e-7)
    og, oo = opt_pair(expansion_order=p, leaf_size_source=6, multipole_acceptance=0.5, error_tolerance=tol,
                      scalar_potential=kind == 1, hessian=kind == 3, nearfield=precision == "f64")
    if precision == "mixed":  # these orders run the FP64 translations on the mixed path too
        if tol is not None and "Relative" in method.__name__:
            pytest.skip("the estimate of the relative methods is in FP32")
        og.precision = L.FMM_PRECISION_MIXED
    out, res = fm.solve_buffers(b, kind, og, ctx=ctx)
    ref = O.fmm(b, kind, oo)
    assert res.n_m2l > 0
    for rows in (slice(3, 7), slice(7, 16)):
        if kind == 3 and rows.start == 3:
            rows = slice(4, 7)
        scale = np.abs(ref["out"][:, rows]).max()
        # the parity bound of the FP64 solve
        np.testing.assert_allclose(out[:, rows], ref["out"][:, rows], rtol=0, atol=1e-10 * scale + 1e-300)
    assert res.p_max == ref["pmax"]


# The M2L kernel depends on the rows of the launch: their number, the longest, and whether they are
# even (the pairs of five of the longest per SM).  One set of bodies per kind of launch.
def rows_of(ctx):
    import torch
    m2l, _ = fm.get_lists(ctx)
    n = np.bincount(m2l[:, 0])
    sm = torch.cuda.get_device_properties(0).multi_processor_count
    return dict(many=(n > 0).sum() >= 4 * sm, few=(n > 0).sum() <= 2 * sm, even=n.sum() >= 5 * sm * n.max(),
                longest=n.max())


LAUNCHES = {
    # sources, targets (0: the sources), leaf size, acceptance, rule, what rows_of has to say
    "even": (8000, 0, 3, 0.9, fm.Barba, dict(many=True, even=True)),
    "uneven": (6000, 0, 2, 0.6, fm.SelfTuningTreeStop, dict(many=True, even=False)),
    "few": (40000, 1500, 10, 0.6, fm.SelfTuningTreeStop, dict(many=False, few=True)),
    "short": (3000, 0, 20, 0.6, fm.SelfTuningTreeStop, dict(many=False)),
}


def launch(ctx, name, kind, p, precision="f64", method=None):
    n, m, leaf, mac, rule, want = LAUNCHES[name]
    b = np.zeros((n, 5 if kind == 1 else 7))
    rng = np.random.default_rng(n)
    b[:, :3] = rng.random((n, 3))
    b[:, 4:] = rng.standard_normal((n, b.shape[1] - 4)) / n
    pos = None if m == 0 else 2 * rng.random((m, 3)) - 0.5
    og, oo = opt_pair(expansion_order=p, leaf_size_source=leaf, multipole_acceptance=mac, error_tolerance=method,
                      scalar_potential=kind == 1, hessian=kind == 3, nearfield=False,
                      interaction_list_method=rule())
    og.precision = L.FMM_PRECISION_MIXED if precision == "mixed" else L.FMM_PRECISION_F64
    out, res = fm.solve_buffers(b, kind, og, pos, ctx=ctx)
    have = rows_of(ctx)
    assert all(bool(have[k]) == v for k, v in want.items()), have
    assert (have["longest"] >= 128) == (name != "short")
    return out, res, lambda: O.fmm(b, kind, oo, target_pos=pos)


def rows(kind):
    return (slice(3, 4), slice(4, 7)) if kind == 1 else (slice(4, 7), slice(7, 16))


@pytest.mark.parametrize("kind", [1, 3])
@pytest.mark.parametrize("p", [4, 5, 6, 7, 8, 9, 10, 11, 12])
@pytest.mark.parametrize("name", list(LAUNCHES))
def test_fixed_orders_of_every_launch(ctx, kind, p, name):
    """FP64, fixed order, far field alone: the parity bound, for every kernel that these launches take."""
    out, res, oracle = launch(ctx, name, kind, p)
    ref = oracle()["out"]
    for r in rows(kind):
        np.testing.assert_allclose(out[:, r], ref[:, r], rtol=0, atol=1e-10 * np.abs(ref[:, r]).max())
    assert res.p_max == p


@pytest.mark.parametrize("method", METHODS[1:], ids=[m.__name__ for m in METHODS[1:]])
@pytest.mark.parametrize("p", [5, 8, 10, 12])
@pytest.mark.parametrize("name", ["even", "uneven", "few"])
def test_error_control_of_every_launch(ctx, method, p, name):
    """FP64 point sources with error control: the pairs' orders and the parity bound."""
    tol = method(3e-6 if "Relative" in method.__name__ else 1e-7)
    out, res, oracle = launch(ctx, name, 1, p, method=tol)
    ref = oracle()
    for r in rows(1):
        np.testing.assert_allclose(out[:, r], ref["out"][:, r], rtol=0, atol=1e-10 * np.abs(ref["out"][:, r]).max())
    assert res.p_max == ref["pmax"] and bool(res.error_success) == ref["error_success"]


@pytest.mark.parametrize("kind", [1, 3])
@pytest.mark.parametrize("p", [4, 5, 6, 7, 8, 9, 10, 11, 12])
@pytest.mark.parametrize("name", list(LAUNCHES))
def test_fp32_translations(ctx, kind, p, name):
    """Mixed, fixed order, against the FP64 one (pinned to the oracle above).  A pair's
    result is some 2 p sums of up to p terms and two rotations, each rounded at 2^-24 of its terms, and the
    errors of the pairs are independent: far below 100 x 2^-24 of the field's norm."""
    mixed, _, _ = launch(ctx, name, kind, p, "mixed")
    f64, _, _ = launch(ctx, name, kind, p)
    for r in rows(kind):
        assert np.linalg.norm(mixed[:, r] - f64[:, r]) <= 100 * 2.0 ** -24 * np.linalg.norm(f64[:, r])
