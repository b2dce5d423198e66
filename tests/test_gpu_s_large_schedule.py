"""The schedule of factors of more than 128 Mi values (4,096-column items, 512-row chunks, 8 rows in flight) against the
host's S^T S: FP64 and FP32, both S kernels, on a 64x32x32 bar (224 M values; the factor built on the host, so that the
host has a copy to apply)."""
import numpy as np
import pytest

from diffphd_b200 import core, scenes

pytestmark = pytest.mark.gpu


def test_large_factor_matches_the_host():
    sc = scenes.cantilever(cells=(64, 32, 32), steps=1)
    d = core.from_scene(sc)
    d.set_factor_build(1)
    b = np.random.default_rng(9).standard_normal(sc.dofs)
    x = d.debug_ainv(b, sc.dt)
    assert not d.factor_built_on_device() and d.s_padded_values() > 128 << 20
    ref = d.debug_host_sts(b, sc.dt)
    scale = np.abs(ref).max()
    assert np.abs(x - ref).max() <= 1e-12 * scale
    for groups in (True, False):
        d.set_s_kernel(groups)
        assert np.array_equal(d.debug_ainv(b, sc.dt), x)
        assert np.abs(d.debug_ainv(b, sc.dt, fp32=True) - ref).max() <= 2e-6 * scale
