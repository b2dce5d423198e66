"""Which route a solve takes, read from the launch counter: the one-kernel loop of small meshes on its side of the limits
(853 nodes, 4,096 samples, S^T chunks of at most 64 rows, FP64, no contact) and the launched loop past each of them; and
the candidate lists of the mixed contact step on both sides of the rule that picks the FP64 S pass (path entries above a
sixth of the factor's values).  The results themselves are compared in the tests of those paths."""
import numpy as np
import pytest

from diffphd_b200 import core, scenes

pytestmark = pytest.mark.gpu
METHOD = "pd_eigen_alg_phd"

CASES = {  # scene, options, S^T chunk rows, one kernel?
    "hex_16x4x4": (lambda: scenes.cantilever(heterogeneous=True), {}, 0, True),
    "hex_8x8x8_4096_samples": (lambda: scenes.cantilever(cells=(8, 8, 8)), {}, 0, True),
    "hex_9x8x8_4608_samples": (lambda: scenes.cantilever(cells=(9, 8, 8)), {}, 0, False),
    "tet_9x7x9_800_nodes": (lambda: scenes.nh_tet_block(cells=(9, 7, 9)), {}, 0, True),
    "tet_9x8x9_900_nodes": (lambda: scenes.nh_tet_block(cells=(9, 8, 9)), {}, 0, False),
    "chunks_of_64": (lambda: scenes.cantilever(heterogeneous=True), {}, 64, True),
    "chunks_of_128": (lambda: scenes.cantilever(heterogeneous=True), {}, 128, False),
    "graph_replayed": (lambda: scenes.cantilever(heterogeneous=True), {"graph_while": 0}, 0, False),
    "mixed": (lambda: scenes.cantilever(heterogeneous=True), {"fp32_bulk": 1}, 0, False),
    "contact": (lambda: scenes.hetero_contact(cells=(4, 4, 4), dx=0.01, height=0.0), {}, 0, False),
}


@pytest.mark.parametrize("name", CASES)
def test_one_kernel_loop_runs_on_its_side_of_the_limits(name):
    make, options, chunk_rows, one_kernel = CASES[name]
    sc = make()
    d = core.from_scene(sc)
    if chunk_rows:
        d.set_st_schedule(chunk_rows, 4)
    opts = dict(sc.options, max_pd_iter=12, rel_tol=1e-14, abs_tol=0.0, verbose=-1, **options)
    d.debug_ainv(sc.q0, sc.dt)
    qn, vn = np.zeros(sc.dofs), np.zeros(sc.dofs)
    before = d.kernel_launches()
    d.PyForward(METHOD, sc.q0, sc.v0 + 0.05, [], sc.f_ext, sc.dt, opts, qn, vn, [])
    launches, iters = d.kernel_launches() - before, int(d.frame_stats()[0][-1])
    if one_kernel:
        assert iters == 12 and launches < iters
    else:
        assert launches > 6 * iters


@pytest.mark.parametrize("every", [True, False])
def test_candidate_lists_on_both_sides_of_the_path_rule(every):
    sc = scenes.contact_drop(cells=(6, 5, 7), height=0.0, steps=5)
    if not every:
        z = sc.q0.reshape(-1, 3)[:, 2]
        sc.plane = (sc.plane[0], np.nonzero(z <= z.min() + 2 * 0.01)[0])
    d = core.from_scene(sc)
    d.debug_ainv(sc.q0, sc.dt)
    entries, _, _ = d.contact_path_stats()
    assert entries > 0
    assert (24 * entries > 4 * d.s_padded_values()) == every
