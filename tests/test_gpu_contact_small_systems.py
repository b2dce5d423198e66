"""The contact step's paths for few active candidates: active systems on both sides of the 64-candidate limit of the
one-CTA solve, and candidate lists that hold every node (S column paths as large as S) against short lists.

Tolerances: frictionless contact has one solution, so two solves of the same active system that stop at a 1e-8 gate
agree to the gate's accuracy (1e-5 of the displacement, the gate times the slow modes' contraction); two candidate
lists with the same active nodes run the same arithmetic up to summation order in FP64 (1e-7 of the displacement),
and in mixed precision to the FP32 S passes' (2e-4, the bound of the mixed contact test)."""
import numpy as np
import pytest

from diffphd_b200 import core, scenes

pytestmark = pytest.mark.gpu
METHOD = "pd_eigen_alg_phd"


def _roll(sc, opts):
    d = core.from_scene(sc)
    q, v, acts = sc.q0.copy(), sc.v0.copy(), []
    for _ in range(sc.steps):
        qn, vn, act = np.zeros(sc.dofs), np.zeros(sc.dofs), []
        d.PyForward(METHOD, q, v, [], sc.f_ext, sc.dt, opts, qn, vn, act)
        q, v = qn, vn
        acts.append(sorted(act))
    return q, acts


@pytest.mark.parametrize("cells, nodes", [((1, 1, 2), 4), ((7, 7, 2), 64), ((8, 7, 2), 72)])
def test_active_systems_around_the_one_cta_limit(cells, nodes):
    sc = scenes.hetero_contact(cells=cells, dx=0.01, steps=4, height=0.0, friction_mu=0.0)
    opts = dict(sc.options, rel_tol=1e-8, max_pd_iter=4000, verbose=-1)
    out = [_roll(sc, dict(opts, ncp_solver=s)) for s in (0, 1)]
    assert len(out[1][1][-1]) == nodes
    assert out[0][1] == out[1][1]
    assert np.abs(out[1][0] - out[0][0]).max() <= 1e-5 * np.abs(out[0][0] - sc.q0).max()


@pytest.mark.parametrize("fp32, tol", [(0, 1e-7), (1, 2e-4)])
def test_every_node_a_candidate_matches_a_short_list(fp32, tol):
    out = []
    for every in (True, False):
        sc = scenes.contact_drop(cells=(6, 5, 7), height=0.0, steps=5)
        sc.v0 = np.tile([0.0, 0.0, -0.4], sc.n)
        if not every:
            z = sc.q0.reshape(-1, 3)[:, 2]
            sc.plane = (sc.plane[0], np.nonzero(z <= z.min() + 2 * 0.01)[0])
        out.append(_roll(sc, dict(sc.options, rel_tol=1e-8, max_pd_iter=4000, fp32_bulk=fp32, verbose=-1)))
    assert any(out[0][1]) and out[0][1] == out[1][1]
    assert np.abs(out[1][0] - out[0][0]).max() <= tol * np.abs(out[0][0] - sc.q0).max()
