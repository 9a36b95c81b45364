"""Code edges taken from the context's sigma-free ones by multiplications: at
sigmas over the floats' range, around every edge, the tables' code equals the
FP64 expression's; and a kick by zero returns the codes it started from, where
the FP64 expressions do."""
import numpy as np
import pytest

from cafproject_gb300 import params as P
from cafproject_gb300 import synth

pytestmark = pytest.mark.gpu

PI_F = np.float32(4.0) * np.arctan(np.float32(1.0))


@pytest.mark.parametrize("izipv", [1, 2])
def test_edges_equal_fp64_expression(izipv):
    from cafproject_gb300 import cube as C

    nvm1 = (1 << (8 * izipv)) - 1
    n = np.arange(1, nvm1 // 2 + 1, dtype=np.float64)
    g = C.CubeGPU(P.CubeParams(nc=16, nnt=1, izipv=izipv))
    rng = np.random.default_rng(11)
    for s in np.float32(np.r_[1e-38, 1e-30, 3e38, 10.0 ** rng.uniform(-4, 2, 8)]):
        e = np.tan((n - 0.5) * np.float64(PI_F) / nvm1) / synth.vcoef(s)
        v = np.concatenate([(e.view(np.int64) + k).view(np.float64) for k in range(-3, 4)])
        v = np.concatenate([v, -v, [0.0, -0.0, np.inf, -np.inf]])
        direct, table = g.codec_check(s, v)
        np.testing.assert_array_equal(direct, table)
    g.close()


@pytest.mark.parametrize("izipv", [1, 2])
def test_zero_kick_codes(izipv):
    """Every code once through decode and encode, by the tables and in FP64."""
    from cafproject_gb300 import cube as C

    lim = 1 << (8 * izipv - 1)
    g = C.CubeGPU(P.CubeParams(nc=16, nnt=1, izipv=izipv))
    for s in np.float32([1e-30, 0.037, 12.0]):
        codes = np.arange(-lim, lim)
        nvm1 = np.float32(2 * lim - 1)
        arg = np.float32(np.float32(PI_F * codes.astype(np.float32)) / nvm1)
        v = np.tan(arg.astype(np.float64)).astype(np.float32).astype(np.float64) / synth.vcoef(s)
        direct, table = g.codec_check(s, v)
        np.testing.assert_array_equal(direct, table)
    g.close()


@pytest.mark.parametrize("izipv", [1, 2])
@pytest.mark.parametrize("fused", [False, True])
def test_idle_particles_keep_their_codes(izipv, fused):
    """Particles alone in their neighbourhood take their code from the table of
    zero kicks: every code through it, in PP's own kick and in the fine kick of
    a fused step without motion, against decode and encode in FP64."""
    from cafproject_gb300 import cube as C

    lim = 1 << (8 * izipv - 1)
    p = P.CubeParams(nc=28, nnt=1, izipv=izipv, pp_on=True, rsoft=0.1)
    n = p.nc ** 3  # one particle to a coarse cell
    codes = np.resize(np.arange(-lim, lim), 3 * n)
    assert 3 * n >= 2 * lim
    nvm1 = np.float32(2 * lim - 1)
    t = np.tan(np.float32(np.float32(PI_F * codes.astype(np.float32)) / nvm1).astype(np.float64)).astype(np.float32)
    g = C.CubeGPU(p)
    for s in np.float32([1e-30, 0.037, 12.0]):
        c = synth.vcoef(s)
        want = np.rint(np.float64(nvm1) * np.arctan(c * (t.astype(np.float64) / c)) / np.float64(PI_F)).astype(np.int64)
        g.upload(np.zeros((n, 3), np.int8 if p.izipx == 1 else np.int16),
                 codes.reshape(n, 3).astype(np.int8 if izipv == 1 else np.int16), np.arange(n, dtype=np.int32),
                 np.ones(n, np.int32), np.zeros((n, 3), np.float32))
        g.set_sigma(s, s)
        g.set_option(C.OPT_PP_FILTER, 2)
        if fused:
            st = g.pp_particle_mesh(0.4, 0.0)[0]
        else:
            st = g.ext_pp_force(0.4, 0.02)
        assert st["npairs"] == n  # each particle its own entry alone: none is active
        np.testing.assert_array_equal(g.download()["vp"].reshape(-1), want)
    g.close()
