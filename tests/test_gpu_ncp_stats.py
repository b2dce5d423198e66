"""The NCP's solve counters (ncp_solver 1) at active systems of either size class: on a block that rests on the ground
every PD iteration has active candidates, so cached solves and fresh factorisations add up to the PD iterations."""
import numpy as np
import pytest

from diffphd_b200 import core, scenes

pytestmark = pytest.mark.gpu
METHOD = "pd_eigen_alg_phd"


@pytest.mark.parametrize("cells, nodes", [((1, 1, 2), 4), ((5, 5, 2), 36), ((7, 7, 2), 64), ((8, 7, 2), 72)])
def test_every_solve_is_counted(cells, nodes):
    sc = scenes.hetero_contact(cells=cells, dx=0.01, steps=4, height=0.0, friction_mu=0.0)
    opts = dict(sc.options, rel_tol=1e-8, max_pd_iter=300, ncp_solver=1, verbose=-1)
    d = core.from_scene(sc)
    q, v, act = sc.q0.copy(), sc.v0.copy(), []
    for _ in range(sc.steps):
        qn, vn, act = np.zeros(sc.dofs), np.zeros(sc.dofs), []
        d.PyForward(METHOD, q, v, [], sc.f_ext, sc.dt, opts, qn, vn, act)
        q, v = qn, vn
    assert len(act) == nodes
    cached, factored, cg_iters, _ = d.ncp_solve_stats(detail=True)
    assert factored > 0
    assert cached + factored == int(np.sum(d.frame_stats()[0]))
    assert (cg_iters > 0) == (cached > 0)
