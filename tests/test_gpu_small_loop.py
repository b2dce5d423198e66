"""The one-kernel loops of small meshes (graph_while 1) against the launched loop (graph_while 0): the same expressions in
the same order, so the same bits, iteration counts and convergence flags, forward and adjoint, over sizes up to the
limits of the one-kernel loop (one block of degrees of freedom, several, ragged ones; one and several rounds of elements)
and past them, Anderson windows 0 to 8, and frames cut off by max_pd_iter."""
import numpy as np
import pytest

from diffphd_b200 import core, scenes

pytestmark = pytest.mark.gpu
METHOD = "pd_eigen_alg_phd"

SCENES = {
    "hex_1x1x1": lambda: scenes.cantilever(cells=(1, 1, 1)),
    "hex_5x2x3": lambda: scenes.cantilever(cells=(5, 2, 3), heterogeneous=True),
    "hex_16x4x4": lambda: scenes.cantilever(heterogeneous=True),
    "hex_16x6x5": lambda: scenes.cantilever(cells=(16, 6, 5), heterogeneous=True),
    "hex_8x8x8": lambda: scenes.cantilever(cells=(8, 8, 8), heterogeneous=True),
    "hex_9x8x8": lambda: scenes.cantilever(cells=(9, 8, 8), heterogeneous=True),
    "tet_2x1x1": lambda: scenes.nh_tet_block(cells=(2, 1, 1)),
    "tet_9x7x9": lambda: scenes.nh_tet_block(cells=(9, 7, 9)),
}


@pytest.mark.parametrize("name", SCENES)
@pytest.mark.parametrize("window, cap", [(5, 60), (0, 7), (1, 40), (8, 40), (5, 1)])
def test_one_kernel_loop_has_the_launched_loops_bits(name, window, cap):
    sc = SCENES[name]()
    rng = np.random.default_rng(1)
    q = sc.q0 + 1e-4 * rng.standard_normal(sc.dofs)
    v = 0.05 * rng.standard_normal(sc.dofs)
    gq, gv = rng.standard_normal(sc.dofs), 0.01 * rng.standard_normal(sc.dofs)
    out = []
    for loop in (1, 0):
        d = core.from_scene(sc)
        opts = dict(sc.options, graph_while=loop, aa_window=window, max_pd_iter=cap, verbose=-1)
        qn, vn = np.zeros(sc.dofs), np.zeros(sc.dofs)
        d.PyForward(METHOD, q, v, [], sc.f_ext, sc.dt, opts, qn, vn, [])
        g = d.backward(METHOD, q, v, [], sc.f_ext, sc.dt, qn, vn, [], gq, gv, opts)
        out.append((qn, vn, g, d.frame_stats()))
    (q1, v1, g1, s1), (q0, v0, g0, s0) = out
    assert np.isfinite(q1).all()
    assert s1[0].tolist() == s0[0].tolist() and s1[1].tolist() == s0[1].tolist() and g1["iters"] == g0["iters"]
    assert np.array_equal(q1, q0) and np.array_equal(v1, v0)
    for key in ("dl_dq", "dl_dv", "dl_df_ext", "dl_dparams", "dl_dstate_p"):
        assert np.array_equal(g1[key], g0[key]), key
