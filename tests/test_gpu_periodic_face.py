"""The boundary's periodic wrap next to the faces: a particle less than half an
ulp below the lower face comes out on the upper bound itself, which is no error,
and keeps its neighbours; one that left the box by more than its length is."""
import numpy as np
import pytest

from gpucell_gb300 import generator as gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_wrap_onto_the_upper_bound(cuda_device, axis):
    from gpucell_gb300 import _lib
    from gpucell_gb300.host import ParticleSystem
    from oracle.binding import Oracle
    f, L = np.float32, 8.0
    rng = np.random.default_rng(axis)
    x = rng.uniform(0, L, (2000, 3)).astype(f)
    x = np.minimum(x, np.nextafter(f(L), f(0)))
    x[:20, axis] = f(-2.0 ** -30)
    x[20:40, axis] = f(L)
    cfg = gen.Config(name="face", bbox=np.array([0, L] * 3, f), pmask=7, n_b1=0, n_b2=0, n_fluid=2000, coor=x,
                     velhalf=np.zeros((2000, 3), f), den_init=2000 / L ** 3, phys=gen.Physics(ext_force=0.0))
    ps, o = ParticleSystem(cfg, noise=False), Oracle(cfg, noise=False)
    _lib.device_status()   # clears
    ps.periodic()
    ps.con_cube_list()
    ps.density()
    o.call("density")
    g = ps.fetch()
    assert _lib.device_status() == 0
    assert (g["pos"][:20, axis] == f(L)).all() and (g["pos"][20:40, axis] == 0).all()
    # about 16 neighbours: a quarter of them in sequence, a dozen roundings each
    np.testing.assert_allclose(g["rho"], o.rho, rtol=(40 / 4 + 16) * 2.0 ** -24)


def test_a_box_length_away_is_reported(cuda_device):
    from gpucell_gb300 import _lib
    from gpucell_gb300.host import ParticleSystem
    cfg = gen.suspension(nx=16, ny=16, nz=16, ncells=0, seed=1)
    ps = ParticleSystem(cfg, noise=False)
    pos = cfg.coor.copy()
    pos[5, 1] += 2.5 * (cfg.bbox[3] - cfg.bbox[2])
    _lib.device_status()
    ps.set_state(pos=pos)
    ps.periodic()
    assert _lib.device_status() == 1
