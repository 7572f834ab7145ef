"""The membrane passes by blocks of triangles: cells of one block, of exactly
full blocks and of many, of different sizes in one system, against the FP64
oracle on deformed cells."""
import numpy as np
import pytest

from gpucell_gb300 import generator as gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("subdivs", [(0,), (2, 0, 3, 1), (4, 1)])
def test_cells_of_several_sizes_match_oracle(cuda_device, subdivs):
    from gpucell_gb300.fused import FusedSystem
    from oracle.binding import Oracle, assert_forces_close
    L = 24.0
    cells = []
    for k, s in enumerate(subdivs):   # 20, 80, 320, 1280, 5120 triangles
        v, f = gen.icosphere(s)
        d = {0: 1.5, 1: 2.0, 2: 3.0, 3: 5.0, 4: 8.0}[s]
        cells.append((gen.biconcave(v, d) + np.array([4.0 + 5.5 * k, 12.0, 11.0 + k]), f))
    rng = np.random.default_rng(8)
    none = np.zeros((0, 3))
    cfg = gen._assemble("cells", [0, L, 0, L, 0, L], 7, none, none, rng.uniform(0, L, (3000, 3)), cells,
                        gen.Physics(ext_force=0.0), 1.0 / 3.0)
    m0 = cfg.n_cell_start
    pos = cfg.coor.copy()   # stretched by up to 3 % from the set-up shape, and shaken
    c = pos[m0:].mean(0)
    pos[m0:] = (pos[m0:] - c) * np.array([1.03, 0.99, 1.01]) + c + rng.uniform(-0.005, 0.005, (cfg.ncp, 3))
    pos = pos.astype(np.float32)
    fs, o = FusedSystem(cfg, noise=False), Oracle(cfg, noise=False)
    o.setup()
    fs.load(pos)
    o.set(pos=pos)
    fs.step(1, 1)
    o.step()
    g = fs.fetch()
    # FP64 sums of FP32 triangles (a few roundings each)
    np.testing.assert_allclose(g["Area64"], o.area, rtol=1e-6)
    np.testing.assert_allclose(g["Vol64"], o.vol, rtol=2e-6)
    np.testing.assert_allclose(g["ParArea"], o.pararea, rtol=2e-6)
    scale = o.force_scale(o.SCALE_MEMB)[m0:]
    assert_forces_close(g["DefForce"], o.defforce, scale, what=str(subdivs))
    assert fs.flags() == 0
    fs.close()
