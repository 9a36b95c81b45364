"""The table-free code certificate and the queues behind it (kicks, re-sort)
against FP64 everywhere, at particle counts around a warp, a block and a
grid-stride pass and in every code width: the same state, bit for bit."""
import numpy as np
import pytest

from cafproject_gb300 import params as P
from cafproject_gb300 import synth

pytestmark = pytest.mark.gpu


def _steps(p, st, exact):
    from cafproject_gb300 import cube as C

    g = C.CubeGPU(p)
    g.upload(st["xp"], st["vp"], st["pid"], st["rhoc"], st["vfield"])
    g.set_sigma(st["sigma_vi"])
    g.set_option(C.OPT_EXACT_KICKS, int(exact))
    for _ in range(2):
        g.update_x(20.0, 30.0, st["vz_max"])
        g.pp_particle_mesh(0.4, 0.05)
    out = g.download()
    g.close()
    return out


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 257, 4097])
@pytest.mark.parametrize("izipx,izipv", [(1, 1), (1, 2), (2, 1), (2, 2)])
def test_queues_equal_fp64(n, izipx, izipv):
    p = P.CubeParams(nc=16, nnt=1, pp_on=True, rsoft=0.1, izipx=izipx, izipv=izipv, np_max=8192)
    st = synth.random_state(p, mean_per_cell=2.5, seed=n, vsig=0.03, clump=3)
    keep = np.zeros(st["xp"].shape[0], bool)
    keep[np.random.default_rng(n).choice(keep.size, size=n, replace=False)] = True
    cell = np.repeat(np.arange(p.nc ** 3), st["rhoc"])
    st["rhoc"] = np.bincount(cell[keep], minlength=p.nc ** 3).astype(np.int32)
    for k in ("xp", "vp", "pid"):
        st[k] = st[k][keep]
    a, b = _steps(p, st, False), _steps(p, st, True)
    for k in a:
        np.testing.assert_array_equal(a[k], b[k])
