"""The list passes with several lanes per particle (small systems) against the
FP64 oracle: one size of each number of lanes, walls of both kinds, and lists
shorter than the lanes (a rarefied gas, some particles without a partner)."""
import numpy as np
import pytest

from gpucell_gb300 import generator as gen

pytestmark = pytest.mark.gpu


def _gas(n, side, seed=2):
    rng = np.random.default_rng(seed)
    x = (rng.uniform(0, 1, (n, 3)) * side).astype(np.float32)
    x[x >= np.float32(side)] = 0.0
    bbox = np.array([0, side] * 3, np.float32)
    return gen.Config(name="gas", bbox=bbox, pmask=7, n_b1=0, n_b2=0, n_fluid=n, coor=x, velhalf=np.zeros_like(x),
                      den_init=1.0, phys=gen.Physics(ext_force=0.0))


@pytest.mark.parametrize("kind", ["gas", "channel 8", "channel 4", "channel 2", "channel 1"])
def test_lanes_match_oracle(cuda_device, kind):
    from gpucell_gb300.fused import FusedSystem
    from oracle.binding import Oracle, assert_forces_close
    if kind == "gas":
        cfg = _gas(700, 11.0)
    else:   # 7 k, 55 k, 104 k and 149 k particles
        k = {"channel 8": 13, "channel 4": 29, "channel 2": 37, "channel 1": 42}[kind]
        cfg = gen.channel(nx=2 * k, ny=k, nz=k + 1, wall_layers=3, b1_layers=1, cell_subdiv=2, cell_diameter=3.0)
    mob = slice(cfg.n_b1 + cfg.n_b2, None)
    fs, o = FusedSystem(cfg, noise=True), Oracle(cfg, noise=True)
    o.setup()
    # one step from rest: both sides evaluate the forces on the same positions
    fs.step(1, 1)
    o.step()
    g = fs.fetch()
    np.testing.assert_array_equal(g["pos"], o.pos.astype(np.float32))
    np.testing.assert_allclose(g["rho"][mob], o.rho[mob], rtol=2e-6)
    assert_forces_close(g["force"][mob], o.force[mob], o.force_scale()[mob], what=kind)
    wall = slice(cfg.n_b1, cfg.n_b1 + cfg.n_b2)
    if cfg.n_b2:
        np.testing.assert_allclose(g["vel"][wall], o.vel[wall], rtol=0, atol=2e-5 * np.abs(o.vel).max())
    assert fs.flags() == 0
    fs.close()
