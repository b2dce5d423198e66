"""The FP32 S^T S pair's error against the FP64 pair, by the factor's size class: the default schedule's longer items and
chunks must not be less accurate than 64-row chunks, whose lanes add eight rows in a row (set_st_schedule(64, 4) sums
every chunk in one run per lane).  Relative L2 error, rms over right-hand sides of white noise and over smooth ones
(A^-1 of noise); one sum per lane over the 256- and 512-row chunks has 1.2 to 2.2 times the error.  5% are left for the
eight right-hand sides of each kind."""
import numpy as np
import pytest

from diffphd_b200 import core, scenes

pytestmark = pytest.mark.gpu

SCENES = {
    "tet_32x16x16": lambda: scenes.nh_tet_block(),                                              # 7 M values
    "hex_24": lambda: scenes.cantilever(cells=(24, 24, 24), steps=1),                           # 19 M
    "hex_48x24x24": lambda: scenes.cantilever(cells=(48, 24, 24), heterogeneous=True, steps=1),  # 54 M
    "hex_64x32x32": lambda: scenes.cantilever(cells=(64, 32, 32), heterogeneous=True, steps=1),  # 224 M
}


def _errors(sc, schedule):
    d = core.from_scene(sc)
    if schedule:
        d.set_st_schedule(*schedule)
    out = {"noise": [], "smooth": []}
    for seed in range(8):
        w = np.random.default_rng(seed).standard_normal(sc.dofs)
        for kind, b in (("noise", w), ("smooth", d.debug_ainv(w, sc.dt))):
            x, y = d.debug_ainv(b, sc.dt), d.debug_ainv(b, sc.dt, fp32=True)
            out[kind].append(np.linalg.norm(y - x) / np.linalg.norm(x))
    return {k: float(np.sqrt(np.mean(np.square(v)))) for k, v in out.items()}


@pytest.mark.parametrize("name", SCENES)
def test_default_schedule_is_as_accurate_as_short_chunks(name):
    sc = SCENES[name]()
    short, default = _errors(sc, (64, 4)), _errors(sc, None)
    for kind in short:
        assert default[kind] <= 1.05 * short[kind], (kind, default, short)
