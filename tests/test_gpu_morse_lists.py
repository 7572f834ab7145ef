"""The Morse lists, built by a warp per vertex: cells of fewer vertices than a
warp, of many more than a warp per cube of the aggregation grid, touching one
another and lying across the faces of a periodic box, against the FP64
oracle's aggregation forces.

Tolerance: 2e-5 of the largest force, as for the aggregation of the channel
(sums of up to a few hundred FP32 terms of a few roundings each)."""
import dataclasses

import numpy as np
import pytest

from gpucell_gb300 import generator as gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("labels", ["runs", "permuted"])
@pytest.mark.parametrize("subdivs, max_cut", [((0, 1, 0), 1.2), ((4, 0, 3), 1.2), ((3, 4, 2, 1), 2.5)])
def test_aggregation_matches_oracle(cuda_device, subdivs, max_cut, labels):
    from gpucell_gb300.fused import FusedSystem
    from oracle.binding import Oracle
    L = 14.0
    cells = []
    for k, s in enumerate(subdivs):   # 12, 42, 162, 642, 2562 vertices
        v, f = gen.icosphere(s)
        # stacked along y a short way apart, the stack across a corner of the box
        cells.append((gen.biconcave(v, 3.0) + np.array([0.4 * k, 1.3 * k - 1.0, 0.3]), f))
    rng = np.random.default_rng(5)
    none = np.zeros((0, 3))
    phys = gen.Physics(ext_force=0.0, sur_energy=5.0, max_cut=max_cut, zero_len=0.3, sca_fac=4.0)
    cfg = gen._assemble("stack", [0, L, 0, L, 0, L], 7, none, none, rng.uniform(0, L, (2000, 3)), cells, phys, 1.0 / 3.0)
    o = Oracle(cfg, noise=False)
    o.setup()
    o.step()
    if labels == "permuted":   # every candidate's label is compared
        perm = np.roll(np.arange(len(subdivs), dtype=np.int32), 1)
        cfg = dataclasses.replace(cfg, celltab=perm[cfg.celltab])
    fs = FusedSystem(cfg, noise=False)
    fs.step(1, 1)
    g = fs.fetch()
    scale = np.abs(o.aggforce).max()
    assert scale > 0
    np.testing.assert_allclose(g["AggForce"], o.aggforce, rtol=0, atol=2e-5 * scale)
    assert fs.flags() == 0
    fs.close()
