"""The paired stencil scatter at particle counts that leave a part of the last
warp's pairs empty (n^3 = 8 or 24 beyond a multiple of 32) and lattices
of one to three cells a particle: the gradient against FP64 autograd."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ng,npd", [(18, 18), (54, 18), (44, 22), (50, 50)])
def test_gradient_at_partial_warps(ng, npd):
    from cafproject_gb300 import dpm as D
    from oracle import dpm_oracle as orc

    sim = D.DiffPM(ng, npd, 9.0, 0.0, 4, ckpt_every=2, box=2.0 * npd)
    filt, green = sim.tables()
    vf = sim.info()["vf"]
    simulate, density = D.autograd_functions()
    target = sim.density(sim.forward(sim.noise(2))[0]).detach()

    n = sim.noise(1).requires_grad_(True)
    x, _ = simulate.apply(n, sim)
    ((density.apply(x, sim) - target) ** 2).sum().backward()

    m = sim.noise(1).double().cpu().requires_grad_(True)
    xo, _ = orc.simulate(m, filt.astype("f8"), green.astype("f8"), ng, npd, vf, sim.drift, sim.kick)
    rho = orc.deposit(xo, ng, npd, float(ng) ** 3 / npd ** 3)
    ((rho - target.double().cpu()) ** 2).sum().backward()
    g, r = n.grad.double().cpu(), m.grad
    # the bound the gradients are held to at whole warps
    assert float((g - r).norm() / r.norm()) < 1e-3
    sim.close()
