"""update_x's sigma_v sums against FP64 over the state it leaves, with the
block partials' number at its smallest, odd, beyond one per thread of the last
pass and at its cap."""
import numpy as np
import pytest

from cafproject_gb300 import params as P
from cafproject_gb300 import synth

pytestmark = pytest.mark.gpu


# particles per cell: nc = 16 has 4096 cells, so 4 blocks; then 37, 300 and 2048
@pytest.mark.parametrize("nc,mean", [(16, 0.5), (16, 9.1), (20, 38.4), (40, 33.0)])
def test_sums_match_fp64(nc, mean):
    from cafproject_gb300 import cube as C

    p = P.CubeParams(nc=nc, nnt=1, pp_on=False, np_max=int(nc ** 3 * mean * 1.1) + 4096)
    st = synth.random_state(p, mean_per_cell=mean, seed=3)
    g = C.CubeGPU(p)
    g.upload(st["xp"], st["vp"], st["pid"], st["rhoc"], st["vfield"])
    g.set_sigma(st["sigma_vi"])
    up = g.update_x(0.0, 0.0, st["vz_max"])
    s = g.download()
    g.close()
    arg = (synth.PI_F * np.arange(-32768, 32768, dtype=np.float32)) / np.float32(65535)
    dec = np.tan(arg.astype(np.float64)).astype(np.float32) / synth.vcoef(st["sigma_vi"])
    v = dec[s["vp"].astype(np.int64) + 32768]
    vf = s["vfield"].astype(np.float64)
    cell = np.repeat(np.arange(nc ** 3), s["rhoc"])
    # float-float accumulators (about 2^-46 a term), FP64 from there on
    assert up["sum_r"] == pytest.approx((v * v).sum(), rel=1e-11)
    assert up["sum_s"] == pytest.approx(((v + vf[cell]) ** 2).sum(), rel=1e-11)
    # the cells' squares are rounded to FP32 first (three products, two sums)
    assert up["sum_c"] == pytest.approx((vf * vf).sum(), rel=5 * 2.0 ** -24)
    assert up["sigma_vi_new"] == pytest.approx(np.sqrt((v * v).sum() / v.shape[0]) / np.sqrt(3.0), rel=1e-6)
