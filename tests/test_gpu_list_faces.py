"""Lists of particles at the periodic faces: less than half an ulp below the
lower one (the wrapped FP32 position is the upper bound itself) and the floats
on either side of both.  The density is the oracle's within FP32 sums (1e-5),
where one missed neighbour of a particle next to it would be a tenth."""
import numpy as np
import pytest

from gpucell_gb300 import generator as gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", ["eight", "one"])
@pytest.mark.parametrize("lo", [0.0, -5.0])
@pytest.mark.parametrize("graph", [False, True])
def test_particles_at_the_faces(cuda_device, lo, lanes, graph):
    from gpucell_gb300.fused import FusedSystem
    from oracle.binding import Oracle
    L, nfluid = (10.0, 3000) if lanes == "eight" else (20.0, 60000)   # lanes per slot of the list build
    f = np.float32
    lo, hi = f(lo), f(lo + L)
    rng = np.random.default_rng(1)
    pos = np.clip(rng.uniform(lo, hi, (nfluid, 3)).astype(f), lo, np.nextafter(hi, lo))
    at = [np.nextafter(hi, lo), np.nextafter(np.nextafter(hi, lo), lo), hi, np.nextafter(hi, f(100)), lo,
          np.nextafter(lo, f(-100)), np.nextafter(lo, hi)]
    if lo == 0:
        at += [f(-2.0 ** -30), f(-2.0 ** -22)]
        assert f(at[-2] + f(L)) == hi
    for axis in range(3):
        rows = rng.choice(nfluid, 60, replace=False)
        pos[rows, axis] = rng.choice(np.array(at, f), 60)
    none = np.zeros((0, 3))
    cfg = gen._assemble("faces", [float(lo), float(hi)] * 3, 7, none, none, pos, [],
                        gen.Physics(ext_force=0.0, dt=1e-6), 1.0 / 3.0)
    assert np.array_equal(cfg.coor, pos)
    o = Oracle(cfg, noise=False)
    o.setup()
    o.step()
    fs = FusedSystem(cfg, noise=False, skin=0.125, graph=graph)
    fs.step(1, 1)
    g = fs.fetch()
    np.testing.assert_allclose(g["rho"], o.rho, rtol=1e-5)
    assert fs.flags() == 0
    fs.close()
