"""k_dest's common case beside the general one: particles at tile and cell faces
(codes 0 and the last), moves up to the buffer depth, one and several tiles;
FP64 everywhere takes the general form for every particle, so the two must
agree to the bit, statistics included."""
import numpy as np
import pytest

from cafproject_gb300 import params as P
from cafproject_gb300 import synth

pytestmark = pytest.mark.gpu


def _step(p, st, exact, dt, vz):
    from cafproject_gb300 import cube as C

    g = C.CubeGPU(p)
    g.upload(st["xp"], st["vp"], st["pid"], st["rhoc"], st["vfield"])
    g.set_sigma(st["sigma_vi"])
    g.set_option(C.OPT_EXACT_KICKS, int(exact))
    stats = g.update_x(dt, dt, vz)
    out = g.download()
    g.close()
    return stats, out


@pytest.mark.parametrize("nc,nnt", [(16, 1), (24, 2), (36, 3)])
@pytest.mark.parametrize("izipx", [1, 2])
@pytest.mark.parametrize("cells", [0.0, 0.4, 2.5, 5.5])
def test_common_case_equals_general(nc, nnt, izipx, cells):
    p = P.CubeParams(nc=nc, nnt=nnt, pp_on=False, izipx=izipx)
    st = synth.random_state(p, mean_per_cell=3.0, seed=nc + izipx, vsig=0.02)
    lo, hi = np.iinfo(p.xdtype).min, np.iinfo(p.xdtype).max
    rng = np.random.default_rng(5)
    face = rng.random(st["xp"].shape) < 0.3
    st["xp"][face] = rng.choice(np.array([0, -1, lo, hi], p.xdtype), size=int(face.sum()))
    vmax = np.abs(st["vfield"]).max() + 8 * st["sigma_vi"]
    dt = np.float32(cells * 4.0 / vmax)  # the fastest particle moves about `cells` coarse cells
    (sa, a), (sb, b) = (_step(p, st, e, dt, float(vmax)) for e in (False, True))
    for k in a:
        np.testing.assert_array_equal(a[k], b[k])
    for k in ("nplocal", "nlost", "ndup", "max_disp", "nlayer", "rank_walked"):
        assert sa[k] == sb[k], k
