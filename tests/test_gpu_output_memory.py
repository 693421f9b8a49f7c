"""Target buffers in memory that is not the context GPU's own: managed memory and another GPU's
(filled by a copy, so that no peer access is needed)."""
import ctypes as C

import numpy as np
import pytest

import fastmultipole_b200 as fm
from fastmultipole_b200 import _lib as L

pytestmark = pytest.mark.gpu

N = 3001


def solve(ctx, bodies, out_ptr, timed):
    """fmm_solve of device bodies into device memory at out_ptr."""
    src = L.SourceSystem(L.FMM_POINT_SOURCE, N, 5, bodies.data_ptr(), L.FMM_MEMORY_DEVICE)
    tgt = L.TargetSystem(N, None, 0, out_ptr, L.FMM_MEMORY_DEVICE)
    opt = fm.make_options(expansion_order=4, leaf_size_source=20, scalar_potential=True)
    res = L.Result()
    ctx.check(L.lib().fmm_solve(ctx.handle, C.byref(tgt), C.byref(src), C.byref(opt), C.byref(res) if timed else None))


@pytest.mark.parametrize("with_result", [True, False])
@pytest.mark.parametrize("where", ["own", "managed", "other GPU"])
def test_target_buffer(where, with_result):
    import torch
    from cuda.bindings import runtime as rt
    if where == "other GPU" and torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    rng = np.random.default_rng(3)
    b = np.zeros((N, 5))
    b[:, :3], b[:, 4] = rng.random((N, 3)), rng.random(N)
    ctx = fm.Context(0)
    opt = fm.make_options(expansion_order=4, leaf_size_source=20, scalar_potential=True)
    ref, _ = fm.solve_buffers(b, L.FMM_POINT_SOURCE, opt, ctx=ctx)  # host buffers
    bodies = torch.from_numpy(b).to("cuda:0")
    torch.cuda.synchronize(0)
    if where == "managed":
        err, ptr = rt.cudaMallocManaged(N * 16 * 8, rt.cudaMemAttachGlobal)
        assert int(err) == 0
        out = np.ctypeslib.as_array(C.cast(int(ptr), C.POINTER(C.c_double)), (N, 16))
        out[:] = -1.0
        solve(ctx, bodies, int(ptr), with_result)
        got = out.copy()
        del out
        rt.cudaFree(ptr)
    else:
        buf = torch.full((N, 16), -1.0, dtype=torch.float64, device="cuda:0" if where == "own" else "cuda:1")
        torch.cuda.synchronize(buf.device)
        solve(ctx, bodies, buf.data_ptr(), with_result)
        got = buf.cpu().numpy()
    np.testing.assert_array_equal(got, ref)
    ctx.close()
