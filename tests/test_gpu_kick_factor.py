"""The kicks on meshes that hold the forces themselves: with the factor
a_mid*dt/6/pi at the limits of the fast path (zero, below the normal floats,
near overflow) the same codes as in FP64 everywhere, and after a fused step the
field calls still return force*a_mid*dt/6/pi, rounded as the kick terms are."""
import numpy as np
import pytest

from cafproject_gb300 import params as P
from cafproject_gb300 import synth

pytestmark = pytest.mark.gpu


def _state(pp_on=False):
    from cafproject_gb300 import cube as C

    p = P.CubeParams(nc=24, nnt=2, pp_on=pp_on, mass_p=8.0)
    st = synth.random_state(p, mean_per_cell=3, seed=5, vsig=0.02, clump=40)

    def make():
        g = C.CubeGPU(p)
        g.upload(st["xp"], st["vp"], st["pid"], st["rhoc"], st["vfield"])
        g.set_sigma(st["sigma_vi"])
        return g

    return C, make


@pytest.mark.parametrize("a_mid,dt", [(0.4, 0.02), (0.4, 0.0), (0.4, -0.5), (1e-20, 1e-18), (0.4, 1e-30), (0.4, 3e-38),
                                      (1.0, 1e15), (1e19, 1e19), (0.4, 1e30)])
@pytest.mark.parametrize("fused", [False, True])
def test_factors_equal_fp64(a_mid, dt, fused):
    C, make = _state()
    out = []
    for exact in (0, 1):
        g = make()
        g.set_option(C.OPT_EXACT_KICKS, exact)
        if fused:
            g.particle_mesh(a_mid, dt)
        else:
            g.fine_forces()
            g.fine_kick(a_mid, dt)
            g.coarse_forces()
            g.coarse_kick(a_mid, dt)
        out.append(g.download()["vp"])
        g.close()
    np.testing.assert_array_equal(out[0], out[1])


def test_fields_after_a_fused_step():
    C, make = _state()
    a_mid, dt = np.float32(0.37), np.float32(0.021)

    def pre(f):
        return (((f * a_mid) * dt) / np.float32(6.0)) / np.float32(np.pi)

    a, b = make(), make()
    a.fine_forces()
    a.coarse_forces()
    b.particle_mesh(float(a_mid), float(dt))
    for field in (C.FIELD_FORCE_F, C.FIELD_FORCE_C):
        raw = a.get_field(field)
        for _ in range(2):  # the same however often it is read
            np.testing.assert_array_equal(b.get_field(field), pre(raw))
    # a field that was written comes back as written, and the next step's are its own
    raw_f = a.get_field(C.FIELD_FORCE_F)
    b.set_field(C.FIELD_FORCE_F, raw_f)
    np.testing.assert_array_equal(b.get_field(C.FIELD_FORCE_F), raw_f)
    b.fine_forces()
    np.testing.assert_array_equal(b.get_field(C.FIELD_FORCE_F), raw_f)
    a.close()
    b.close()


@pytest.mark.parametrize("scale", [1.0, 1e13, 1e17, np.inf, np.nan])
def test_written_forces_equal_fp64(scale):
    """Stage kicks on force meshes that the caller wrote, and on those that a
    fused step left, with and without the exact option."""
    C, make = _state()
    out = []
    for exact in (0, 1):
        g = make()
        g.set_option(C.OPT_EXACT_KICKS, exact)
        g.particle_mesh(0.4, 0.02)
        g.fine_kick(0.4, 0.02)
        g.coarse_kick(0.4, 0.02)
        for field, kick in ((C.FIELD_FORCE_F, g.fine_kick), (C.FIELD_FORCE_C, g.coarse_kick)):
            f = g.get_field(field)
            f.reshape(-1)[::97] *= np.float32(scale)
            g.set_field(field, f)
            kick(0.3, 0.01)
        out.append(g.download()["vp"])
        g.close()
    np.testing.assert_array_equal(out[0], out[1])
