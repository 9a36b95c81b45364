"""The fixed-point sums of the differentiable form's deposit turned into its
padded FP32 mesh, at row lengths around the warp's stretch of cells (64), and
their zeroing: a second density of other positions must not see the first's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ng,npd", [(16, 16), (18, 18), (62, 31 * 2), (64, 32), (66, 22), (130, 26), (300, 20)])
def test_density_rows_against_fp64(ng, npd):
    import torch

    from cafproject_gb300 import dpm as D
    from oracle import dpm_oracle as O

    sim = D.DiffPM(ng, npd, 9.0, 8.0, 1, box=float(ng))
    mass = float(ng) ** 3 / npd ** 3
    for seed in (1, 2):
        x = torch.randn(npd ** 3, 3, generator=torch.Generator().manual_seed(seed)) * 2.0
        rho = sim.density(x.cuda()).cpu().double()
        xd = x.double()
        ref = O.deposit(xd, ng, npd, mass)
        # a weight's three products and the mass round at most five times, the
        # fractions once each; the sum is exact up to its one rounding
        terms = torch.zeros(ng ** 3, dtype=torch.float64)
        for idx, _ in O._corners(xd, ng, npd):
            terms.index_add_(0, idx, torch.ones(idx.shape[0], dtype=torch.float64))
        bound = 2.0 ** -24 * (8 * mass * terms.view(ng, ng, ng) + ref)
        assert bool(((rho - ref).abs() <= bound).all())
        assert np.isclose(rho.sum(), float(ng) ** 3, rtol=1e-6)
    sim.close()
