"""FP64 y = S v by row groups against one warp per row segment (the same per-lane order: the same bits) and against the
host's S^T S, on factors on both sides of the schedule's size limits: rows of one segment and of several
2,048-column ones."""
import numpy as np
import pytest

from diffphd_b200 import core, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [lambda: scenes.cantilever(cells=(3, 1, 2), steps=1),
                                  lambda: scenes.nh_tet_block(cells=(13, 9, 11)),
                                  lambda: scenes.nh_tet_block(),
                                  lambda: scenes.cantilever(cells=(24, 24, 24), steps=1)],
                         ids=["hex_3x1x2", "tet_13x9x11", "tet_32x16x16", "hex_24"])
def test_fp64_row_groups(make):
    sc = make()
    d = core.from_scene(sc)
    b = np.random.default_rng(5).standard_normal(sc.dofs)
    d.debug_ainv(b, sc.dt)
    xs = []
    for groups in (True, False, True):
        d.set_s_kernel(groups)
        xs.append(d.debug_ainv(b, sc.dt))
    assert np.array_equal(xs[0], xs[1]) and np.array_equal(xs[0], xs[2])
    ref = d.debug_host_sts(b, sc.dt)
    assert np.abs(xs[0] - ref).max() <= 1e-12 * np.abs(ref).max()
