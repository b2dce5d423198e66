"""The allocation-free A^-1 entry point at the limit of its scratch array and inside a captured graph.

A 64x32x32 bar needs more than the 32 MiB array with the default 64-row S^T chunks and less with 512-row ones: the
call is refused in the first case and served in the second.  The captured call follows a copy and a join with another
stream (its first kernel is launched with programmatic serialization) and must repeat the plain call's bits.
"""
import ctypes as C

import numpy as np
import pytest

from diffphd_b200 import core, scenes

pytestmark = pytest.mark.gpu


def _call(d, sc, db, dx, stream):
    return core.load_library().dphd_ainv_noalloc(d._h, C.c_double(sc.dt), C.c_void_p(db.data_ptr()),
                                                 C.c_void_p(dx.data_ptr()), 0, C.c_void_p(stream.cuda_stream))


@pytest.mark.parametrize("chunk_rows, accepted", [(0, False), (512, True)])
def test_scratch_limit_follows_the_callers_chunks(chunk_rows, accepted):
    import torch
    sc = scenes.cantilever(cells=(64, 32, 32), steps=1)
    d = core.from_scene(sc)
    if chunk_rows:
        d.set_st_schedule(chunk_rows, 8)
    b = np.random.default_rng(3).standard_normal(sc.dofs)
    ref = d.debug_ainv(b, sc.dt)
    db = torch.as_tensor(b, device="cuda")
    dx = torch.zeros_like(db)
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    rc = _call(d, sc, db, dx, st)
    st.synchronize()
    assert (rc == 0) == accepted
    if accepted:
        assert np.array_equal(dx.cpu().numpy(), ref)
    else:
        assert b"bytes of scratch" in core.load_library().dphd_last_error()


def test_captured_call_after_a_copy_and_a_join():
    import torch
    sc = scenes.nh_tet_block(cells=(8, 4, 4), dx=0.01, steps=1)
    d = core.from_scene(sc)
    rng = np.random.default_rng(4)
    bs = [rng.standard_normal(sc.dofs) for _ in range(2)]
    refs = [d.debug_ainv(b, sc.dt) for b in bs]
    src = torch.zeros(sc.dofs, dtype=torch.float64, device="cuda")
    db, dx, other = torch.zeros_like(src), torch.zeros_like(src), torch.zeros_like(src)
    st, side = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    assert _call(d, sc, db, dx, st) == 0  # looks the scratch address up
    st.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        side.wait_stream(st)
        with torch.cuda.stream(side):
            other.copy_(src)
        db.copy_(src)
        st.wait_stream(side)
        assert _call(d, sc, db, dx, st) == 0
        db.add_(other)
        assert _call(d, sc, db, dx, st) == 0
    for b, ref in zip(bs, refs):
        src.copy_(torch.as_tensor(b))
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(dx.cpu().numpy(), 2 * ref)  # doubling is exact
