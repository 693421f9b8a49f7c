"""Targets without a position (a NaN coordinate) get NaN in every requested row, whether or not the
far field has a translation to make, and leave the other targets alone."""
import numpy as np
import pytest

import fastmultipole_b200 as fm
from fastmultipole_b200 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,hess", [(1, False), (1, True), (3, False), (3, True)])
@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("n", [40, 4000])
@pytest.mark.parametrize("phi", [False, True])
def test_nan_target(kind, hess, precision, n, phi):
    rng = np.random.default_rng(6)
    b = np.zeros((n, 5 if kind == 1 else 7))
    b[:, :3], b[:, 4:] = rng.random((n, 3)), rng.standard_normal((n, b.shape[1] - 4))
    pos = rng.random((n, 3))
    opt = fm.make_options(expansion_order=4, leaf_size_source=20, scalar_potential=phi, hessian=hess,
                          precision=precision)
    ctx = fm.Context(0)
    ref, _ = fm.solve_buffers(b, kind, opt, pos, ctx=ctx)
    pos[3, 1] = np.nan
    out, res = fm.solve_buffers(b, kind, opt, pos, ctx=ctx)
    assert (res.n_m2l > 0) == (n > 40)
    rows = ([3] if phi else []) + [4, 5, 6] + (list(range(7, 16)) if hess else [])
    assert np.all(np.isnan(out[3, rows]))
    others = np.delete(np.arange(n), 3)
    assert np.all(np.isfinite(out[others]))
    if n == 40:
        assert np.all(abs(out[others][:, rows] - ref[others][:, rows]) <= 1e-4 * abs(ref[:, rows]).max())
    ctx.close()
