"""The cube sweep of the boundary entry points where its blocks can go wrong:
cubes with more particles than a block takes at once, stencils with more
candidates than are staged at once, periodic axes of three cubes, sparse grids
(several cubes per block, most of them empty), and positions that the caller
has not wrapped into the box.  Compared with the FP64 oracle.
"""
import numpy as np
import pytest

from gpucell_gb300 import generator as gen

pytestmark = pytest.mark.gpu

U = 2.0 ** -24   # FP32 unit roundoff


def _config(kind, seed=3):
    """Random particles (Bound1, Bound2, fluid) in a fully periodic box."""
    rng = np.random.default_rng(seed)
    box, n = {"crowded": ((3.25, 4.25, 3.5), 4000), "sparse": ((41.0, 17.0, 23.0), 900),
              "clump": ((9.0, 8.0, 11.0), 2600), "odd": ((3.1, 7.9, 5.2), 3001)}[kind]
    box = np.array(box)
    x = rng.uniform(0, 1, (n, 3)) * box
    if kind == "clump":   # most of them within one cube, the rest anywhere
        x[600:] = np.array([4.4, 3.4, 10.9]) + rng.uniform(-0.45, 0.45, (n - 600, 3))
    x = np.round(np.mod(x, box) * 1024) / 1024
    x = rng.permutation(x).astype(np.float32)
    x = np.where(x >= box, x - box, x).astype(np.float32)
    nb = n // 10
    phys = gen.Physics(ext_force=0.0)
    bbox = np.stack([np.zeros(3), box], 1).ravel().astype(np.float32)
    return gen.Config(name=kind, bbox=bbox, pmask=7, n_b1=nb, n_b2=nb, n_fluid=n - 2 * nb, coor=x,
                      velhalf=np.zeros((n, 3), np.float32), den_init=float(n / box.prod()), phys=phys)


@pytest.mark.parametrize("kind", ["crowded", "sparse", "clump", "odd"])
def test_sweeps_match_oracle(cuda_device, kind):
    from gpucell_gb300.host import ParticleSystem
    from oracle.binding import Oracle, assert_forces_close
    cfg = _config(kind)
    rng = np.random.default_rng(5)
    vel = rng.normal(size=(cfg.n, 3)).astype(np.float32).astype(np.float64)
    ps, o = ParticleSystem(cfg, noise=True), Oracle(cfg, noise=True)
    ps.set_state(vel=vel)
    o.set(vel=vel)
    count = o.neighbor_stats()[0].max()
    # a lane adds at most a quarter of the terms (each good to about a dozen roundings) in sequence
    rtol = (count / 4 + 16) * U
    fluid = slice(cfg.n_b1 + cfg.n_b2, None)
    ps.density()
    o.call("density")
    g = ps.fetch()
    np.testing.assert_allclose(g["rho"][fluid], o.rho[fluid], rtol=rtol)
    o.set(rho=g["rho"])
    ps.bound2_vel()
    o.call("bound2_vel")
    g = ps.fetch()
    wall = slice(cfg.n_b1, cfg.n_b1 + cfg.n_b2)
    # weighted means of velocities up to 5: the weights and the products round as above
    np.testing.assert_allclose(g["vel"][wall], o.vel[wall], rtol=0, atol=2 * 5 * rtol)
    np.testing.assert_array_equal(g["vel"][fluid], vel[fluid].astype(np.float32))
    ps.eos()
    g = ps.fetch()
    o.set(vel=g["vel"], press=g["press"])
    ps.sdpd_force()
    o.call("sdpd_force")
    g = ps.fetch()
    assert not g["force"][:cfg.n_b1 + cfg.n_b2].any()
    assert_forces_close(g["force"], o.force, o.force_scale(o.SCALE_SDPD), k=16 + count / 4, what=f"{kind} sdpd")
    ps.set_state(force=np.zeros((cfg.n, 3)))
    o.set(force=np.zeros((cfg.n, 3)))
    ps.rep_force()
    o.call("rep_force")
    g = ps.fetch()
    assert_forces_close(g["force"], o.force, o.force_scale(o.SCALE_REP), k=64 + count / 4, what=f"{kind} repulsion")


@pytest.mark.parametrize("kind", ["odd", "sparse"])
def test_unwrapped_positions(cuda_device, kind):
    """A caller may leave positions somewhat outside the box (a step's motion,
    not wrapped yet): every sweep takes their minimum image (coordinates and
    box lengths are multiples of 2^-10 here, so the shift itself is exact)."""
    from gpucell_gb300.host import ParticleSystem
    cfg = _config(kind)
    L = np.round((cfg.bbox[1::2]) * 1024) / 1024
    cfg.bbox[1::2] = L
    x = np.where(cfg.coor >= L, cfg.coor - L, cfg.coor).astype(np.float32)
    rng = np.random.default_rng(9)
    loose = rng.random((cfg.n, 3)) < 0.3
    shift = 1.0 * (loose & (x < 0.4)) - 1.0 * (loose & (x > L - 0.4))
    out = []
    for pos in (x, x + shift * L):
        ps = ParticleSystem(cfg, noise=False)
        ps.set_state(pos=pos.astype(np.float32), vel=rng.normal(size=(cfg.n, 3)) * 0 + 1.0)
        ps.con_cube_list()
        ps.density()
        ps.eos()
        ps.sdpd_force()
        out.append(ps.fetch())
    a, b = out
    fluid = slice(cfg.n_b1 + cfg.n_b2, None)
    np.testing.assert_allclose(b["rho"][fluid], a["rho"][fluid], rtol=2 * 100 * U)
    scale = np.abs(a["press"]).max() / a["rho"].min() ** 2 * 67.0 * 100
    np.testing.assert_allclose(b["force"], a["force"], rtol=0, atol=scale * 2 * 100 * U * 20)


@pytest.mark.parametrize("ncells,subdiv", [(1, 2), (7, 1), (40, 2)])
def test_aggregation_matches_oracle(cuda_device, ncells, subdiv):
    """From one cell (no pair) to forty interpenetrating ones in a box of
    seven cubes: more vertices in a cube and in a stencil than a block takes
    at once, stencils across every periodic face."""
    from gpucell_gb300.host import ParticleSystem
    from oracle.binding import Oracle, assert_forces_close
    phys = gen.Physics(ext_force=0.0, sur_energy=3.0e-3, sca_fac=1.5, zero_len=0.3, max_cut=2.5)
    rng = np.random.default_rng(ncells)
    L = 7.25
    verts, faces = gen.icosphere(subdiv)
    shape = gen.biconcave(verts, 3.0)
    cells = [(shape @ gen.random_rotation(rng).T + rng.uniform(0, L, 3) * 0.999, faces) for _ in range(ncells)]
    fluid = rng.uniform(0, L, (2000, 3))
    none = np.zeros((0, 3))
    cfg = gen._assemble("packed", [0, L, 0, L, 0, L], 7, none, none, fluid, cells, phys, 1.0 / 3.0)
    ps, o = ParticleSystem(cfg, noise=False), Oracle(cfg, noise=False)
    o.setup()
    wrapped = np.mod(cfg.coor, np.float32(L)).astype(np.float32)
    o.set(pos=wrapped)
    ps.set_state(pos=wrapped)
    ps.con_cube_list()
    area = ps.d["ParArea"].cpu().numpy()
    o.set(pararea=area)
    z = np.zeros((cfg.n, 3))
    ps.set_state(force=z)
    o.set(force=z)
    ps.agg_force()
    o.call("agg_force")
    g = ps.fetch()
    s = o.force_scale(o.SCALE_MORSE)
    # e^{beta (r0 - r)} of a rounded argument up to 3.3, squared, and the sum over the lanes
    k = 64 + cfg.ncp / 8
    assert_forces_close(g["force"], o.force, s, k=k, what="aggregation")
    assert_forces_close(g["AggForce"], o.aggforce, s[cfg.n_cell_start:], k=k, what="aggregation per vertex")
    assert ncells == 1 or np.abs(o.aggforce).max() > 0
