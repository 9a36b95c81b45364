"""The scan of the cell counts at one chunk (4096), a ragged one, the largest
size of the one-launch form (2^17 counts) and beyond it: a re-sort without any
motion must leave every particle where it is."""
import numpy as np
import pytest

from cafproject_gb300 import params as P
from cafproject_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,mean", [(16, 0.02), (16, 3.0), (18, 5.0), (50, 1.5), (52, 1.5), (64, 0.7)])
def test_resort_without_motion(nc, mean):
    from cafproject_gb300 import cube as C

    p = P.CubeParams(nc=nc, nnt=1, pp_on=False)
    st = synth.random_state(p, mean_per_cell=mean, seed=nc, clump=4)
    g = C.CubeGPU(p)
    g.upload(st["xp"], st["vp"], st["pid"], st["rhoc"], st["vfield"])
    g.set_sigma(st["sigma_vi"])
    up = g.update_x(0.0, 0.0, st["vz_max"])
    out = g.download()
    g.close()
    assert up["nplocal"] == st["pid"].size
    for k in ("rhoc", "pid", "xp"):
        np.testing.assert_array_equal(out[k], st[k])


@pytest.mark.parametrize("nc", [16, 52])  # one launch, three launches
def test_count_sum_does_not_wrap(nc):
    # neighbouring counts that exceed the particle count by 2^32 in all, in the
    # last chunk: refused like any other wrong sum
    from cafproject_gb300 import cube as C

    p = P.CubeParams(nc=nc, nnt=1, pp_on=False)
    st = synth.random_state(p, mean_per_cell=1.0, seed=nc)
    bad = st["rhoc"].copy()
    last = bad.reshape(-1)[-16:]
    last[1:4] += np.array([2 ** 31 - 100, 2 ** 31 - 100, 200], np.int32)
    assert bad.astype(np.int64).sum() == st["pid"].size + 2 ** 32 and bad.min() >= 0
    g = C.CubeGPU(p)
    with pytest.raises(C.CubeError) as e:
        g.upload(st["xp"], st["vp"], st["pid"], bad, st["vfield"])
    assert e.value.code == 6
    g.close()
