"""Lists built from positions outside the box: a particle is sorted by its cell
before the wrap, whose rounding can put the wrapped position into the next
cell.  It must neither list itself nor miss a neighbour: the density is the
oracle's within FP32 sums (1e-5), where an entry for the particle itself would
add W(0), a tenth of it."""
import numpy as np
import pytest

from gpucell_gb300 import generator as gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("nfluid", [3000, 60000])   # several lanes per slot, and one thread per slot
def test_wrapped_onto_a_cell_boundary(cuda_device, axis, nfluid):
    from gpucell_gb300.fused import FusedSystem
    from oracle.binding import Oracle
    L, n = np.float32(20.0 if nfluid > 50000 else 10.0), 35 if nfluid > 50000 else 17   # cells of the lists
    rng = np.random.default_rng(axis)
    pos = rng.uniform(0, L, (nfluid, 3)).astype(np.float32)
    special = pos[:600, axis]
    special[:] = (rng.integers(1, n, 600) * (float(L) / n) - float(L)).astype(np.float32)
    special += (rng.integers(-3, 4, 600) * np.float32(2.0 ** -21)).astype(np.float32)
    invw = np.float32(n / float(L))
    before = np.floor(special * invw).astype(int) % n
    after = np.floor((special + L) * invw).astype(int) % n
    assert (before != after).any()
    none = np.zeros((0, 3))
    cfg = gen._assemble("outside", [0, float(L)] * 3, 7, none, none, pos, [],
                        gen.Physics(ext_force=0.0, dt=1e-6), 1.0 / 3.0)
    o = Oracle(cfg, noise=False)
    o.setup()
    o.step()
    fs = FusedSystem(cfg, noise=False, skin=0.125)
    fs.step(1, 1)
    g = fs.fetch()
    np.testing.assert_allclose(g["rho"], o.rho, rtol=1e-5)
    assert fs.flags() == 0
    fs.close()
