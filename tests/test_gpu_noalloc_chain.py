"""Calls of the allocation-free A^-1 entry point one behind the other on one stream, each on the result of the one before
(d_b of a call is d_x of the last, no kernel in between), against the same calls with a synchronisation after each: the
first kernel of a call is launched while the last one of the call before drains, and must not read its b early."""
import ctypes as C

import numpy as np
import pytest

from diffphd_b200 import core, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("cells", [(2, 2, 2), (8, 4, 4), (24, 12, 12)])
def test_chained_calls_read_the_result_of_the_call_before(cells, fp32):
    import torch
    sc = scenes.nh_tet_block(cells=cells, dx=0.01, steps=1)
    d = core.from_scene(sc)
    b = np.random.default_rng(7).standard_normal(sc.dofs)
    d.debug_ainv(b, sc.dt)  # builds the factor
    L = core.load_library()
    st = torch.cuda.Stream()

    def call(src, dst):
        rc = L.dphd_ainv_noalloc(d._h, C.c_double(sc.dt), C.c_void_p(src.data_ptr()), C.c_void_p(dst.data_ptr()), fp32,
                                 C.c_void_p(st.cuda_stream))
        assert rc == 0, L.dphd_last_error().decode()

    x0 = torch.as_tensor(b, device="cuda")
    links = 4
    ref = [x0] + [torch.zeros_like(x0) for _ in range(links)]
    for i in range(links):
        torch.cuda.synchronize()
        call(ref[i], ref[i + 1])
    torch.cuda.synchronize()
    assert all(float(r.abs().max()) > 0 for r in ref)
    got = [[x0] + [torch.zeros_like(x0) for _ in range(links)] for _ in range(25)]
    inplace = x0.clone()
    torch.cuda.synchronize()
    for xs in got:
        for i in range(links):
            call(xs[i], xs[i + 1])
    for _ in range(links):
        call(inplace, inplace)
    torch.cuda.synchronize()
    for xs in got:
        assert all(torch.equal(a, r) for a, r in zip(xs, ref))
    assert torch.equal(inplace, ref[-1])
