"""Morse pairs that come within MaxCut between two list builds: at the build
they are more than two widths of MaxCut/2 cubes apart, with two cubes between
them, but nearer than MaxCut + skin.  Against the FP64 oracle's aggregation
forces while the lists are still those; 1e-3 of the largest force (FP32
positions in a box of 23 move e^{2 beta r} and the areas by 1e-5; a missed
pair is all of the force)."""
import dataclasses

import numpy as np
import pytest

from gpucell_gb300 import generator as gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("cubes", [18, 6])   # 6: MaxCut fits three times into the box, MaxCut + skin does not
def test_pairs_that_approach_are_listed(cuda_device, axis, cubes):
    from gpucell_gb300.fused import FusedSystem
    from oracle.binding import Oracle
    L = 68 / 3 if cubes == 18 else 7.6
    w = L / cubes
    verts, faces = gen.icosphere(0)
    pole = verts[0] / np.linalg.norm(verts[0])
    e = np.eye(3)[axis]
    v = pole + e   # half-turn that takes the pole to e
    verts = 0.4 * (2 * np.outer(verts @ v, v) / (v @ v) - verts)
    other = [a for a in range(3) if a != axis]
    cells, vel = [], []
    for k in range(16 if cubes == 18 else 1):
        at = np.zeros(3)
        at[other[0]], at[other[1]] = 1.5 + 5.6 * (k % 4), 1.5 + 5.6 * (k // 4)
        c = (k + cubes - 2) % cubes   # the pairs also lie across the faces
        cells += [(verts + at + e * ((c + 1) * w - 0.02 - 0.4), faces), (-verts + at + e * ((c + 3) * w + 0.02 + 0.4), faces)]
        vel += [e * 500.0] * 12 + [-e * 500.0] * 12
    none = np.zeros((0, 3))
    phys = gen.Physics(ext_force=0.0, dt=1e-5, sur_energy=5.0, max_cut=2.5, zero_len=0.3, sca_fac=1.5)
    cfg = gen._assemble("poles", [0, L] * 3, 7, none, none, none, cells, phys, 1.0 / 3.0)
    cfg = dataclasses.replace(cfg, den_init=3.5, coor=np.mod(cfg.coor, np.float32(L)).astype(np.float32))
    vel = np.array(vel)
    o = Oracle(cfg, noise=False)
    o.setup()
    o.set(vel=vel)
    fs = FusedSystem(cfg, noise=False, skin=0.125)
    fs.load(cfg.coor, vel, cfg.velhalf)
    for _ in range(10):
        o.step()
    fs.step(1, 1)   # builds the lists of the loaded state
    builds = fs.stats()["rebuilds"]
    fs.step(9, 1)
    assert fs.stats()["rebuilds"] == builds
    g = fs.fetch()
    scale = np.abs(o.aggforce).max()
    assert scale > 0
    np.testing.assert_allclose(g["AggForce"], o.aggforce, rtol=0, atol=1e-3 * scale)
    assert fs.flags() == 0
    fs.close()


@pytest.mark.parametrize("box, skin", [((10.01, 12.0, 11.0), 1.0), ((7.6, 9.0, 7.7), 0.3)])
def test_boxes_of_few_cubes(cuda_device, box, skin):
    """Boxes that take MaxCut, or five times half of it, along every axis but not
    MaxCut + skin."""
    from gpucell_gb300.fused import FusedSystem
    from oracle.binding import Oracle
    max_cut = 4.0 if box[0] > 10 else 2.5
    rng = np.random.default_rng(2)
    verts, faces = gen.icosphere(1)
    cells = [(1.2 * verts + rng.uniform(0, 1, 3) * box, faces) for _ in range(6)]
    none = np.zeros((0, 3))
    phys = gen.Physics(ext_force=0.0, dt=1e-6, sur_energy=5.0, max_cut=max_cut, zero_len=0.3, sca_fac=1.5)
    cfg = gen._assemble("few", np.stack([np.zeros(3), box], 1).ravel(), 7, none, none, rng.uniform(0, 1, (500, 3)) * box,
                        cells, phys, 1.0 / 3.0)
    o = Oracle(cfg, noise=False)
    o.setup()
    fs = FusedSystem(cfg, noise=False, skin=skin)
    for _ in range(2):
        o.step()
    fs.step(2, 1)
    g = fs.fetch()
    scale = np.abs(o.aggforce).max()
    assert scale > 0
    # sums of up to 200 FP32 terms of a few roundings each, as for the cells of the other tests
    np.testing.assert_allclose(g["AggForce"], o.aggforce, rtol=0, atol=2e-5 * scale)
    assert fs.flags() == 0
    fs.close()
