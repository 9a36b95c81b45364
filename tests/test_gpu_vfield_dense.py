"""The velocity means of cells around the thread, warp and block limits (24 and
256 particles, stretches of 32 and 256) against the visit-order walker, which
sums every cell in one thread."""
import numpy as np
import pytest

from cafproject_gb300 import params as P
from cafproject_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("izipv", [1, 2])
@pytest.mark.parametrize("vbulk", [0.0, 0.05])
def test_dense_cells_match_the_walker(izipv, vbulk):
    from cafproject_gb300 import cube as C

    p = P.CubeParams(nc=16, nnt=1, pp_on=False, izipv=izipv, np_max=1 << 17)
    rng = np.random.default_rng(3)
    counts = rng.poisson(6.0, p.nc ** 3).astype(np.int32)
    sizes = [24, 25, 32, 33, 64, 65, 255, 256, 257, 288, 511, 512, 513, 3000]
    counts[rng.choice(counts.size, size=len(sizes), replace=False)] = sizes
    n = int(counts.sum())
    sigma = np.float32(0.01)
    st = dict(xp=rng.integers(-128, 128, size=(n, 3)).astype(p.xdtype),
              vp=synth.encode(rng.normal(0.0, float(sigma), (n, 3)), sigma, izipv).astype(p.vdtype),
              pid=np.arange(n, dtype=np.int32), rhoc=counts,
              vfield=(rng.normal(0.0, 0.02, (p.nc ** 3, 3)) + vbulk).astype(np.float32))
    out = []
    for walk in (0, 1):
        g = C.CubeGPU(p)
        g.upload(**st)
        g.set_sigma(sigma)
        g.set_option(C.OPT_RANK_WALK, walk)
        up = g.update_x(2.0, 2.0, 0.2)
        assert up["rank_walked"] == walk
        out.append(g.download())
        g.close()
    for k in out[0]:
        np.testing.assert_array_equal(out[0][k], out[1][k])
