"""Mesh sizes on both sides of the batched inverse transform and of the maxima
pass's rows per block: the forces against the Green's multiply in FP64, and the
maximum against the forces themselves, fine and coarse."""
import numpy as np
import pytest

from cafproject_gb300 import params as P
from cafproject_gb300 import synth

pytestmark = pytest.mark.gpu


def _max_f2(f):
    a, b, c = f
    return ((a * a + b * b).astype(np.float32) + c * c).max()


# nf = 4 nc: 64 .. 224 batched, 232 not; the coarse meshes are batched throughout
@pytest.mark.parametrize("nc", [16, 18, 34, 56, 58])
def test_forces_and_maxima(nc):
    from cafproject_gb300 import cube as C

    p = P.CubeParams(nc=nc, nnt=1, pp_on=False)
    st = synth.random_state(p, mean_per_cell=3.0, seed=nc, clump=2)
    g = C.CubeGPU(p)
    g.upload(st["xp"], st["vp"], st["pid"], st["rhoc"], st["vfield"])
    for density, forces, rho_id, f_id, k_id, key in (
            (g.fine_density, g.fine_forces, C.FIELD_RHO_F, C.FIELD_FORCE_F, C.FIELD_KERN_F, "f2_max_fine"),
            (g.coarse_density, g.coarse_forces, C.FIELD_RHO_C, C.FIELD_FORCE_C, C.FIELD_KERN_C, "f2_max_coarse")):
        density()
        rho = g.get_field(rho_id).astype(np.float64)
        stats = forces()
        f, kern = g.get_field(f_id), g.get_field(k_id).astype(np.float64)
        spec = np.fft.rfftn(rho)
        for d in range(3):
            ref = np.fft.irfftn(1j * kern[d] * spec, s=rho.shape, axes=(0, 1, 2))
            # FP32 transforms both ways: the parity tests' bar
            assert np.linalg.norm(f[d] - ref) <= 1e-5 * np.linalg.norm(ref)
        assert np.float32(stats[key]) == _max_f2(f)
    g.close()
