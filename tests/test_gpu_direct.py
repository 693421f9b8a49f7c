"""direct! at the edges of its target blocks and source splits, against extended-precision sums."""
import numpy as np
import pytest

import fastmultipole_b200 as fm
from fastmultipole_b200 import _lib as L
import ctypes as C
from test_gpu_nearfield import EPS, bodies, sums

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = fm.Context(0)
    yield c
    c.close()


def direct(ctx, b, kind, pos, hess, precision):
    out = np.zeros((len(pos), 16))
    pos = np.ascontiguousarray(pos)
    src = L.SourceSystem(kind, len(b), b.shape[1], b.ctypes.data, L.FMM_MEMORY_HOST)
    tgt = L.TargetSystem(len(pos), pos.ctypes.data, 3, out.ctypes.data, L.FMM_MEMORY_HOST)
    ctx.check(L.lib().fmm_direct(ctx.handle, C.byref(tgt), C.byref(src), 1, 1, int(hess), precision))
    return out


@pytest.mark.parametrize("kind,hess", [(1, False), (3, False), (3, True)])
@pytest.mark.parametrize("nt,ns", [(1, 1), (1, 5000), (3, 129), (257, 128), (512, 1023), (513, 127), (1025, 513)])
@pytest.mark.parametrize("mixed", [False, True])
def test_blocks_and_splits(ctx, kind, hess, nt, ns, mixed):
    b = bodies(ns, kind, 1.0, 21)
    pos = np.concatenate([b[::5, :3], bodies(nt, 1, 1.0, 22)[:, :3]])[:nt]  # some on sources
    out = direct(ctx, b, kind, pos, hess, L.FMM_PRECISION_MIXED if mixed else L.FMM_PRECISION_F64)
    r = np.linalg.norm(pos[:, None] - b[None, :, :3], axis=2)
    far = np.abs(b[:, :3]).max() + np.abs(pos).max()
    for cols, ref in zip((slice(3, 4), slice(4, 7), slice(7, 16)), sums(pos, b, hess)):
        if ref is None:
            continue
        got = out[:, cols].reshape(np.shape(ref[0]))
        tol = 4 * (ns + 16) * EPS * ref[1]
        if mixed:
            # FP32 coordinates relative to a target of the block: an error of 2^-24 of their size, i.e.
            # 2^-24 far / r of the pair's distance, times the order of the kernel (<= 5); the terms'
            # roundings and a chunk of 128 FP32 additions
            near = np.where(r > 0, r, np.inf).min(1)
            rel = 2.0 ** -24 * (150 + 5 * 4 * far / near)
            tol = tol + (rel if got.ndim == 1 else rel[:, None]) * ref[1]
        assert np.all(np.isfinite(got))
        assert np.all(abs(got - ref[0]) <= tol)


@pytest.mark.parametrize("kind,hess", [(1, False), (3, False), (3, True)])
@pytest.mark.parametrize("mixed", [False, True])
def test_pairs_without_a_distance_are_left_out(ctx, kind, hess, mixed):
    """A pair counts if r^2 > 0: bodies with a NaN coordinate, and the own infinite or NaN strength of
    a coincident body, add nothing (to the other targets they do)."""
    prec = L.FMM_PRECISION_MIXED if mixed else L.FMM_PRECISION_F64
    b = bodies(700, kind, 1.0, 23)
    pos = bodies(300, 1, 1.0, 24)[:, :3]
    rows = slice(3, 16) if hess else slice(3, 7)
    bad = b.copy()
    bad[[5, 129, 699], [0, 1, 2]] = np.nan
    b[[5, 129, 699], 4:] = 0.0
    got, ref = direct(ctx, bad, kind, pos, hess, prec), direct(ctx, b, kind, pos, hess, prec)
    tol = 1e-4 if mixed else 1e-12  # another path sums the same terms
    assert np.all(np.isfinite(got[:, rows]))
    np.testing.assert_allclose(got[:, rows], ref[:, rows], rtol=0, atol=tol * np.abs(ref[:, rows]).max())
    # a target without a position: no pair at all
    pos[17, 1] = np.nan
    got = direct(ctx, bad, kind, pos, hess, prec)
    assert np.all(got[17, rows] == 0) and np.all(np.isfinite(np.delete(got, 17, 0)[:, rows]))
    # a body of infinite strength on a target: only that target leaves it out
    pos[40] = bad[300, :3]
    bad[300, 4:] = np.inf
    got = direct(ctx, bad, kind, pos, hess, prec)
    assert np.all(np.isfinite(got[40, rows])) and not np.any(np.all(np.isfinite(np.delete(got, [17, 40], 0)[:, 4:7]), 1))
