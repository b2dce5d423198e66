"""The line between the one-CTA solve of small active systems and the grid's cached-factor solve (56 active candidates):
which of the two ran on either side of it, from the solve counters, and the result against a fresh factorisation at every
PD iteration (ncp_solver 0).  Frictionless contact has one solution, so two solves that stop at a 1e-8 gate agree to the
gate's accuracy: 1e-5 of the displacement."""
import numpy as np
import pytest

from diffphd_b200 import core, scenes

pytestmark = pytest.mark.gpu
METHOD = "pd_eigen_alg_phd"


def _roll(sc, opts):
    d = core.from_scene(sc)
    q, v, act = sc.q0.copy(), sc.v0.copy(), []
    for _ in range(sc.steps):
        qn, vn, act = np.zeros(sc.dofs), np.zeros(sc.dofs), []
        d.PyForward(METHOD, q, v, [], sc.f_ext, sc.dt, opts, qn, vn, act)
        q, v = qn, vn
    return q, sorted(act), d.ncp_solve_stats()


@pytest.mark.parametrize("cells, nodes, one_cta", [((10, 4, 2), 55, True), ((7, 6, 2), 56, True), ((18, 2, 2), 57, False),
                                                   ((7, 7, 2), 64, False)])
def test_line_of_the_one_cta_solve(cells, nodes, one_cta):
    sc = scenes.hetero_contact(cells=cells, dx=0.01, steps=4, height=0.0, friction_mu=0.0)
    opts = dict(sc.options, rel_tol=1e-8, max_pd_iter=4000, verbose=-1)
    q0, a0, s0 = _roll(sc, dict(opts, ncp_solver=0))
    q1, a1, (cached, factored) = _roll(sc, dict(opts, ncp_solver=1))
    assert s0 == (0, 0)
    assert len(a1) == nodes and a0 == a1
    assert factored > 0 and (cached == 0) == one_cta
    assert np.abs(q1 - q0).max() <= 1e-5 * np.abs(q0 - sc.q0).max()
