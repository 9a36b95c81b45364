"""Local ranks of the counting re-sort, found within warps of particles in
storage order: cells that cross one or several warps, up to the size listed for
a block of their own, and part-filled warps give the visit-order walker's state."""
import numpy as np
import pytest

from cafproject_gb300 import params as P
from cafproject_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,mean", [(1, 1.0), (31, 1.0), (33, 1.0), (257, 1.0), (4097, 2.0), (20001, 6.0),
                                    (120000, 33.0), (400000, 100.0)])
def test_counting_path_equals_walker(n, mean):
    from cafproject_gb300 import cube as C

    p = P.CubeParams(nc=16, nnt=1, pp_on=False, np_max=600000)
    st = synth.random_state(p, mean_per_cell=mean, seed=n, vsig=0.02, clump=0)
    np0 = st["xp"].shape[0]
    if n < np0:
        keep = np.zeros(np0, bool)
        keep[np.random.default_rng(n).choice(np0, size=n, replace=False)] = True
        cell = np.repeat(np.arange(p.nc ** 3), st["rhoc"])
        st["rhoc"] = np.bincount(cell[keep], minlength=p.nc ** 3).astype(np.int32)
        for k in ("xp", "vp", "pid"):
            st[k] = st[k][keep]
    out = []
    for path in (0, 1):
        g = C.CubeGPU(p)
        g.upload(st["xp"], st["vp"], st["pid"], st["rhoc"], st["vfield"])
        g.set_sigma(st["sigma_vi"])
        g.set_option(C.OPT_RANK_WALK, path)
        u = g.update_x(2.0, 3.0, st["vz_max"])
        assert u["rank_walked"] == path and u["max_disp"] <= 1
        out.append(g.download())
        g.close()
    for k in ("xp", "vp", "pid", "rhoc", "vfield"):
        np.testing.assert_array_equal(out[0][k], out[1][k])
