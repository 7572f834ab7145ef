"""The force pass where the fluid lies far above the rest density of the equation
of state (a stiff gas), there and at it, with one lane per particle and with
several, half velocities too: against the FP64 oracle's forces from the GPU's
own densities, per particle |dF_i| <= 1e-5 |F_i| + 16 u S_i."""
import dataclasses

import pytest

from gpucell_gb300 import generator as gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rest", [1e-6, 1e-3, 0.1, 0.6])
@pytest.mark.parametrize("nx", [24, 64])   # eight lanes per particle, and one
@pytest.mark.parametrize("sound2", [20.0, 30.0])
def test_forces_far_above_the_rest_density(cuda_device, rest, nx, sound2):
    from gpucell_gb300.fused import FusedSystem
    from oracle.binding import Oracle, assert_forces_close
    cfg = gen.suspension(nx=nx, ny=nx, nz=nx, ncells=1, subdiv=2, seed=3)
    cfg = dataclasses.replace(cfg, den_init=cfg.den_init * rest,
                              phys=dataclasses.replace(cfg.phys, dt=1e-20, sound2=sound2))
    o = Oracle(cfg, noise=False)
    o.setup()
    o.step()
    fs = FusedSystem(cfg, noise=False)
    fs.step(1, 1)
    g = fs.fetch()
    o.forces_from_density(g["rho"], g["press"])
    assert_forces_close(g["force"], o.force, o.force_scale(31))
    assert fs.flags() == 0
    fs.close()
