"""What the allocation-free entry point says when it refuses a mesh: the byte count and the schedule that it is counted for
(not the factor's own one, which needs less), and a way out that works."""
import ctypes as C
import re

import numpy as np
import pytest

from diffphd_b200 import core, scenes

pytestmark = pytest.mark.gpu


def test_refusal_names_the_schedule_it_counts():
    import torch
    sc = scenes.cantilever(cells=(64, 32, 32), steps=1)
    b = np.random.default_rng(3).standard_normal(sc.dofs)
    db = torch.as_tensor(b, device="cuda")
    dx = torch.zeros_like(db)
    L = core.load_library()

    def call(d):
        rc = L.dphd_ainv_noalloc(d._h, C.c_double(sc.dt), C.c_void_p(db.data_ptr()), C.c_void_p(dx.data_ptr()), 0, None)
        torch.cuda.synchronize()
        return rc

    d = core.from_scene(sc)
    d.debug_ainv(b, sc.dt)
    assert call(d) != 0
    message = L.dphd_last_error().decode()
    found = re.search(r"(\d+) bytes of scratch, counted for 2,048-column items and S\^T chunks of (\d+) rows", message)
    assert found and int(found[1]) > 32 << 20 and int(found[2]) == 64
    assert "dphd_debug_set_st_schedule" in message
    d.set_st_schedule(512, 8)
    ref = d.debug_ainv(b, sc.dt)
    assert call(d) == 0
    assert np.array_equal(dx.cpu().numpy(), ref)
