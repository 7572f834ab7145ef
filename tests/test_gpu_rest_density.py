"""The pressure term of the force pass at densities near the rest density, at
half of it and without one, with one and two sound speeds, against the FP64
oracle: per particle |dF_i| <= 1e-5 |F_i| + 16 u S_i, from the oracle's own
densities and from the GPU's."""
import dataclasses

import pytest

from gpucell_gb300 import generator as gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rest", [1.0, 2.0, 0.0])
@pytest.mark.parametrize("sound2", [20.0, 30.0])
def test_forces_at_rest_density(cuda_device, rest, sound2):
    from gpucell_gb300.fused import FusedSystem
    from oracle.binding import Oracle, assert_forces_close
    cfg = gen.suspension(nx=24, ny=24, nz=24, ncells=1, subdiv=2, seed=3)
    cfg = dataclasses.replace(cfg, den_init=cfg.den_init * rest,
                              phys=dataclasses.replace(cfg.phys, dt=1e-20, sound2=sound2))
    o = Oracle(cfg, noise=False)
    o.setup()
    o.step()
    fs = FusedSystem(cfg, noise=False)
    fs.step(1, 1)
    g = fs.fetch()
    mov = slice(cfg.n_b1 + cfg.n_b2, cfg.n)
    assert_forces_close(g["force"][mov], o.force[mov], o.force_scale()[mov])
    o.forces_from_density(g["rho"], g["press"])
    assert_forces_close(g["force"][mov], o.force[mov], o.force_scale(31)[mov])
    assert fs.flags() == 0
    fs.close()
