"""The power spectrum's binning at row lengths around a warp (ng/2 + 1 modes: 9,
33, 35, 64 and 65) against the oracle, auto and cross, and twice the same."""
import numpy as np
import pytest

from cafproject_gb300 import params as P
from cafproject_gb300 import synth

pytestmark = pytest.mark.gpu

O = pytest.importorskip("oracle.cube_oracle")


@pytest.mark.parametrize("nc,mult", [(16, 1), (16, 4), (34, 2), (126, 1), (32, 4)])
def test_rows_against_oracle(nc, mult):
    from cafproject_gb300 import cube as C

    p = P.CubeParams(nc=nc, nnt=1, pp_on=False, box=3.0 * nc)
    st = synth.random_state(p, mean_per_cell=2.0, seed=nc + mult, clump=5)
    ng = mult * nc
    g = C.CubeGPU(p)
    g.upload(st["xp"], st["vp"], st["pid"], st["rhoc"], st["vfield"])
    xg, again = g.power_spectrum(ng, p.box), g.power_spectrum(ng, p.box)
    cross = g.power_spectrum(ng, p.box, delta2=O.cic_density(p, st["xp"], st["rhoc"], ng))
    g.close()
    np.testing.assert_array_equal(xg, again)
    xo = O.power_spectrum(p, st["xp"], st["rhoc"], ng, p.box)
    np.testing.assert_array_equal(xg[:, 0], xo[:, 0])
    full = xo[:, 0] > 0
    # the existing bars: FP32 transform and sums against the oracle's
    np.testing.assert_allclose(xg[full, 1], xo[full, 1], rtol=1e-6)
    np.testing.assert_allclose(xg[full, 2], xo[full, 2], rtol=1e-4)
    np.testing.assert_allclose(xg[full, 5:7], xo[full, 5:7], rtol=1e-5)
    np.testing.assert_allclose(cross[full, 2], xg[full, 2], rtol=1e-6)
    np.testing.assert_allclose(cross[full, 3:5], np.repeat(xo[full, 2:3], 2, 1), rtol=2e-4)
