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


@pytest.mark.parametrize("room", [0, 1])
@pytest.mark.parametrize("path", [0, 1, 2])
def test_one_particle_lands_in_two_tiles(room, path):
    """A particle that ends within 2^-50 of a cell behind its tile's face: in
    its own tile's frame the sum rounds onto the face, in the next tile's it
    stays behind it, and both tiles get a copy (update_particle.f90:69).  With
    arrays for one particle less the step is refused and the state is kept."""
    from cafproject_gb300 import cube as C

    sigma, dt, code = np.float32(0.02153819613158703), np.float32(0.12764865159988403), 20000
    PI_F = np.float32(4.0) * np.arctan(np.float32(1.0))
    arg = np.float32(np.float32(PI_F * np.float32(code)) / np.float32(65535))
    dx = np.float64(dt) * (np.float64(np.float32(np.tan(np.float64(arg)))) / synth.vcoef(sigma)) * 0.25
    off = 255.5 / 256
    assert np.ceil((11 + off) + dx) == 12 and np.ceil((-1 + off) + dx) == 1  # the two frames, nt = 12

    n = 40
    p = P.CubeParams(nc=24, nnt=2, pp_on=False, np_max=n + room)
    rhoc = np.zeros(p.nc ** 3, np.int32)
    rhoc[11] = n  # tile 0, cell (12, 1, 1): the last along x
    xp, vp = np.zeros((n, 3), p.xdtype), np.zeros((n, 3), p.vdtype)
    xp[7, 0], vp[7, 0] = -1, code  # the last of the 256 positions in a cell
    st = dict(xp=xp, vp=vp, pid=np.arange(1, n + 1, dtype=np.int32), rhoc=rhoc,
              vfield=np.zeros((p.nc ** 3, 3), np.float32))
    g = C.CubeGPU(p)
    g.upload(**st)
    g.set_sigma(sigma)
    g.set_option(C.OPT_RANK_WALK, path)
    if not room:
        with pytest.raises(C.CubeError) as e:
            g.update_x(dt, dt, 1.0)
        assert "np_max" in str(e.value)
        out = g.download()
        for k in ("xp", "vp", "pid", "rhoc"):
            np.testing.assert_array_equal(out[k].reshape(-1), st[k].reshape(-1))
    else:
        s = g.update_x(dt, dt, 1.0)
        assert s["ndup"] == 1 and s["nplocal"] == n + 1
        out = g.download()
        # the next tile's first cell along x, the second tile's cell 0
        assert out["rhoc"].reshape(-1)[11] == n and out["rhoc"].reshape(-1)[12 ** 3] == 1
        np.testing.assert_array_equal(np.sort(out["pid"]), np.sort(np.r_[st["pid"], 8]))
        assert out["pid"][-1] == 8
    g.close()
