"""The cached-factor NCP solve's grid reductions: its partial sums of p.w and of r.r follow each other without a barrier
between the total of the first and the stores of the second, so they have slots of their own.  A frame solved again and
again from the same state (hundreds of conjugate-gradient iterations a frame) gives the same bits, PD iterations and
CG iterations every time; active systems of one to five 64-row tiles, with and without friction."""
import numpy as np
import pytest

from diffphd_b200 import core, scenes

pytestmark = pytest.mark.gpu
METHOD = "pd_eigen_alg_phd"


@pytest.mark.parametrize("cells, nodes", [((8, 7, 2), 72), ((12, 12, 3), 169), ((16, 16, 2), 289)])
@pytest.mark.parametrize("mu", [0.0, 0.5])
def test_a_frame_repeats_bit_for_bit(cells, nodes, mu):
    import torch
    sc = scenes.hetero_contact(cells=cells, dx=0.01, steps=1, height=0.0, friction_mu=mu)
    opts = dict(sc.options, rel_tol=1e-8, max_pd_iter=60, ncp_solver=1, verbose=-1)
    d = core.from_scene(sc)
    q = torch.as_tensor(sc.q0, dtype=torch.float64, device="cuda")
    v, f = torch.zeros_like(q), torch.zeros_like(q)
    seen, stats = [], []
    for _ in range(30):
        d.reset_warm_start()
        qn, vn = torch.empty_like(q), torch.empty_like(q)
        before = np.array(d.ncp_solve_stats(detail=True))
        d.forward_device(METHOD, q, v, f, sc.dt, opts, qn, vn)
        stats.append((np.array(d.ncp_solve_stats(detail=True)) - before).tolist() + [int(d.frame_stats()[0][-1])])
        seen.append((qn, vn, d.contact_lambda().clone()))
    assert int((seen[0][2] > 0).sum()) == nodes
    assert stats[0][2] > 0
    assert all(s == stats[0] for s in stats)
    for other in seen[1:]:
        assert all(torch.equal(a, b) for a, b in zip(seen[0], other))
